// One instance of the bit-plane sketch kernels (shm_sketch_bits.cuh): k =
// SKB_K, ASCII and packed reads. The Makefile builds an object per k.
#include <mutex>

#include "shm_prims.cuh"
#include "shm_sketch_bits.cuh"

namespace shm {

template <int K>
void launch_sketch_bits_k(const SketchArgs& a, const SketchTabs* tabs, cudaStream_t s) {
    const bool pk = a.pk_codes != nullptr;
    const int smem = (int)(pk ? sizeof(SkbShared<K, true>) : sizeof(SkbShared<K, false>));
    {  // the dynamic shared memory limit, once per device and kernel
        static std::mutex mu;
        static bool done[2][64] = {};
        int dev = 0;
        SHM_CUDA(cudaGetDevice(&dev));
        std::lock_guard<std::mutex> g(mu);
        if (dev < 0 || dev >= 64) throw shm_cuda_error(cudaErrorInvalidDevice);
        if (!done[pk][dev]) {
            if (pk) SHM_CUDA(cudaFuncSetAttribute(k_sketch_bits<K, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
            else SHM_CUDA(cudaFuncSetAttribute(k_sketch_bits<K, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
            done[pk][dev] = true;
        }
    }
    // tiles of the launch (the first starts at most 63 bases before the reads), a warp each at least
    const size_t n_tiles = (size_t)((a.base1 - a.base0 + 63) / SKB_TILE + 1);
    const int grid = grid_for(n_tiles, SKB_WARPS, pk ? skb_ctas<K, true>() : skb_ctas<K, false>());
    if (pk) k_sketch_bits<K, true><<<grid, SKB_WARPS * 32, smem, s>>>(a, tabs);
    else k_sketch_bits<K, false><<<grid, SKB_WARPS * 32, smem, s>>>(a, tabs);
    SHM_CUDA(cudaGetLastError());
    count_launch();
}
template void launch_sketch_bits_k<SKB_K>(const SketchArgs&, const SketchTabs*, cudaStream_t);

}  // namespace shm
