// One instance of the bit-plane sketch kernels (shm_sketch_bits.cuh): k =
// SKB_K; ASCII and packed reads, and sequences in order. The Makefile builds an object per k.
#include <mutex>

#include "shm_prims.cuh"
#include "shm_sketch_bits.cuh"

namespace shm {

// CTAs of a launch over the sequences of a: every warp at least a tile where
// there are enough (the first tile starts at most 63 bases before them).
template <int K>
int sketch_bits_grid(const SketchArgs& a, bool pk) {
    const size_t n_tiles = (size_t)((a.base1 - a.base0 + 63) / SKB_TILE + 1);
    return grid_for(n_tiles, SKB_WARPS, pk ? skb_ctas<K, true>() : skb_ctas<K, false>());
}

template <int K, bool PK, bool ORD>
static void launch_one(const SketchArgs& a, const SketchTabs* tabs, cudaStream_t s) {
    const int smem = (int)sizeof(SkbShared<K, PK>);
    {  // the dynamic shared memory limit, once per device and kernel
        static std::mutex mu;
        static bool done[64] = {};
        int dev = 0;
        SHM_CUDA(cudaGetDevice(&dev));
        std::lock_guard<std::mutex> g(mu);
        if (dev < 0 || dev >= 64) throw shm_cuda_error(cudaErrorInvalidDevice);
        if (!done[dev]) {
            SHM_CUDA(cudaFuncSetAttribute(k_sketch_bits<K, PK, ORD>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
            done[dev] = true;
        }
    }
    k_sketch_bits<K, PK, ORD><<<sketch_bits_grid<K>(a, PK), SKB_WARPS * 32, smem, s>>>(a, tabs);
    SHM_CUDA(cudaGetLastError());
    count_launch();
}

// Returns the warps of an ordered launch (tabs null: asked for only).
template <int K>
int launch_sketch_bits_k(const SketchArgs& a, const SketchTabs* tabs, cudaStream_t s) {
    if (a.ord_cnt) {
        if (tabs) launch_one<K, false, true>(a, tabs, s);
        return sketch_bits_grid<K>(a, false) * SKB_WARPS;
    }
    if (a.pk_codes) launch_one<K, true, false>(a, tabs, s);
    else launch_one<K, false, false>(a, tabs, s);
    return 0;
}
template int launch_sketch_bits_k<SKB_K>(const SketchArgs&, const SketchTabs*, cudaStream_t);

}  // namespace shm
