// Host-side objects behind the C ABI (context, index, batch scratch).
#pragma once
#include <cuda_runtime.h>
#include <cstdio>
#include <cstdlib>
#include <stdint.h>

#include <string>
#include <vector>

#include "../../include/shmap_gpu.h"
#include "shm_common.cuh"
#include "shm_sketch.cuh"

namespace shm {

uint64_t h_thres(double h_frac);  // src/sketch.rs:126-132

// Sets the message shm_last_error() returns on this thread.
void set_last_error(const std::string& m);

// A device buffer that only grows; released by the destructor.
template <class T>
struct DevBuf {
    T* p = nullptr;
    size_t cap = 0;  // elements
    // Grows (never shrinks). Queued work may still use the old buffer, so a
    // growth waits for the device first; a buffer that grows again takes a
    // quarter more than asked, so that batches of varying size (a server's)
    // stop growing it soon.
    void reserve(size_t n) {
        if (n <= cap && p) return;
        if (p) {
            SHM_CUDA(cudaDeviceSynchronize());
            SHM_CUDA(cudaFree(p));
            n += n / 4;
        }
        if (std::getenv("SHMAP_HOSTPROF"))
            std::fprintf(stderr, "[shmap-host] grow %zu -> %zu bytes\n", cap * sizeof(T), n * sizeof(T));
        p = nullptr;
        size_t want = n < 16 ? 16 : n;
        SHM_CUDA(cudaMalloc(&p, want * sizeof(T)));
        cap = want;
    }
    void release() {
        if (p) cudaFree(p);
        p = nullptr;
        cap = 0;
    }
    ~DevBuf() { release(); }
    DevBuf() = default;
    DevBuf(const DevBuf&) = delete;
    DevBuf& operator=(const DevBuf&) = delete;
};

// Memory of the current device, usable on stream s and, once s has been
// synchronized, on any: from the device's pool (shm_prims.cu) up to POOL_MOST
// bytes, above that from cudaMalloc (the pool keeps less than large builds need
// and would map their memory again after every synchronize: an index of 3.1
// Gbp took 0.61 s with its 3.1 GB of bases in the pool, 0.33 s without).
// pool_put gives it back behind the work queued on s.
constexpr size_t POOL_MOST = (size_t)1 << 28;
void* pool_get(size_t bytes, cudaStream_t s);
inline void pool_put(void* p, size_t bytes, cudaStream_t s) {
    if (bytes > POOL_MOST) cudaFree(p);  // (waits for the device)
    else cudaFreeAsync(p, s);
}
// The bytes of the pool that objects hold for long (PoolBuf) changed by delta:
// what the pool keeps of freed memory comes on top of them.
void pool_live(int64_t delta);

// A temporary of work queued on one stream: given back on that stream, behind
// its last use.
template <class T>
struct TmpBuf {
    T* p = nullptr;
    size_t bytes = 0;
    cudaStream_t s = nullptr;
    void reserve(size_t n, cudaStream_t st) {
        release();
        s = st;
        bytes = n * sizeof(T);
        p = (T*)pool_get(bytes, st);
    }
    void release() {
        if (p) pool_put(p, bytes, s);
        p = nullptr;
    }
    ~TmpBuf() { release(); }
    TmpBuf() = default;
    TmpBuf(const TmpBuf&) = delete;
    TmpBuf& operator=(const TmpBuf&) = delete;
};

// An array of an object that outlives the call that made it and is read on any
// stream: given back when the device is idle (as cudaFree would wait for).
template <class T>
struct PoolBuf {
    T* p = nullptr;
    size_t bytes = 0;
    void reserve(size_t n, cudaStream_t s) {
        if (p) throw shm_cuda_error(cudaErrorInvalidValue);  // made once
        bytes = n * sizeof(T);
        p = (T*)pool_get(bytes, s);
        if (bytes <= POOL_MOST) pool_live((int64_t)bytes);
    }
    ~PoolBuf() {
        if (!p) return;
        cudaDeviceSynchronize();
        pool_put(p, bytes, nullptr);
        if (bytes <= POOL_MOST) try {
                pool_live(-(int64_t)bytes);
            } catch (...) {  // (the driver is gone)
            }
    }
    PoolBuf() = default;
    PoolBuf(const PoolBuf&) = delete;
    PoolBuf& operator=(const PoolBuf&) = delete;
};

// An event for waits (no timing) of one call.
struct StreamEvent {
    cudaEvent_t e = nullptr;
    StreamEvent() { SHM_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming)); }
    ~StreamEvent() { cudaEventDestroy(e); }
    StreamEvent(const StreamEvent&) = delete;
    StreamEvent& operator=(const StreamEvent&) = delete;
};

struct IndexStorage {
    DevIndex dev{};
    PoolBuf<uint32_t> seg_off, key_off, hits, hit_fw, dir, ref_rs;
    PoolBuf<int32_t> seg_sz;
    PoolBuf<uint64_t> ref_h, keys;
    PoolBuf<uint4> btab;
    std::vector<std::string> names;
    std::vector<int32_t> seg_len;        // bases
    std::vector<uint32_t> h_seg_off;     // k-mer offsets (n_seg+1)
    shm_index_stats stats{};
    int32_t k = 0;
    double h_frac = 0;
    int32_t max_matches = -1;
    int device = 0;
    uint32_t max_list = 0;  // longest hit list of the index
};

// An index written to a file and read back (shm_index.cu); failures throw
// IndexFileError with a message.
struct IndexFileError {
    std::string what;
};
void save_index(const IndexStorage* ix, const char* path);
IndexStorage* load_index(const char* path, cudaStream_t s);
// The checks load_index makes, on the host alone (no device is touched).
void check_index_file(const char* path);

// Pinned staging for copies from pageable host memory, one a context (see
// shm_upload.cu), and the copy: dst holds the bytes once s has reached this
// point; pageable src may be changed on return, pinned src once s has got there.
struct UploadStage;
UploadStage* upload_stage_create();
void upload_stage_destroy(UploadStage* u);
void upload(UploadStage* u, int device, void* dst, const void* src, size_t bytes, cudaStream_t s);

// The segments' bases are read from h_seq (host) or, when d_seq is given,
// from device memory (d_seq + seg_off[i], 32 readable bytes past the end).
// luts: the tables of k (create_device_luts).
IndexStorage* build_index(const uint8_t* h_seq, const int64_t* seg_off, int32_t n_seg,
                          const std::vector<std::string>& names, int32_t k, double h_frac, int32_t max_matches,
                          const SketchLuts* luts, UploadStage* up, cudaStream_t s, const uint8_t* d_seq = nullptr);

}  // namespace shm

// The opaque handles of the C ABI.
struct shm_index {
    shm::IndexStorage* s;
};
