// Host bytes in ordinary (pageable) memory on their way to the device. The
// driver's own copy from such memory goes through its staging buffers on the
// calling thread; here the packing threads fill a context's pinned slots and
// queue each slot's copy, so the bytes go up as fast as several cores read
// them. Bytes that are pinned already are copied from where they lie.
//
// The copy takes this way from 64 MiB on, where both take the same time when
// the bytes are in the cores' caches (4.9 and 4.7 ms on 16 cores); for more
// bytes than those hold the threads are faster (240 MiB 24.7 and 11.0 ms), for
// fewer the driver is (16 MiB 1.1 and 1.7 ms: the threads have to wake, and a
// slot's copy costs a call). Slots of 256 KiB took 17 ms for 256 MiB, of 1 MiB
// 12: the queueing calls of all threads take turns.
#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstring>
#include <deque>
#include <mutex>
#include <vector>

#include "shm_internal.hpp"
#include "../host/pack.hpp"

namespace shm {

constexpr size_t UPLOAD_SLOT = (size_t)2 << 20;  // bytes
constexpr size_t UPLOAD_SLOTS = 8;               // 16 MiB a context, made when first needed
constexpr size_t UPLOAD_LEAST = (size_t)64 << 20;

struct UploadStage {
    std::mutex use;  // one upload at a time
    uint8_t* pinned = nullptr;
    std::vector<cudaEvent_t> ev;  // slot's last copy
    // the slots no thread is filling, the longest queued first
    std::mutex mu;
    std::condition_variable cv;
    std::deque<int> idle;
    ~UploadStage() {
        for (cudaEvent_t e : ev)
            if (e) cudaEventDestroy(e);
        if (pinned) cudaFreeHost(pinned);
    }
    bool ready() {
        if (pinned && ev.size() == UPLOAD_SLOTS) return true;
        if (!pinned && cudaHostAlloc((void**)&pinned, UPLOAD_SLOT * UPLOAD_SLOTS, cudaHostAllocDefault) != cudaSuccess) {
            cudaGetLastError();
            pinned = nullptr;
            return false;
        }
        while (ev.size() < UPLOAD_SLOTS) {
            cudaEvent_t e = nullptr;
            if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
                cudaGetLastError();
                return false;
            }
            idle.push_back((int)ev.size());
            ev.push_back(e);
        }
        return true;
    }
};

UploadStage* upload_stage_create() { return new UploadStage(); }
void upload_stage_destroy(UploadStage* u) { delete u; }

void upload(UploadStage* u, int device, void* dst, const void* src, size_t bytes, cudaStream_t s) {
    if (!bytes) return;
    bool staged = u && bytes >= UPLOAD_LEAST;
    if (staged) {
        cudaPointerAttributes a{};
        if (cudaPointerGetAttributes(&a, src) != cudaSuccess) cudaGetLastError();
        else staged = a.type == cudaMemoryTypeUnregistered;
    }
    std::unique_lock<std::mutex> one;
    if (staged) {
        one = std::unique_lock<std::mutex>(u->use);
        staged = u->ready();
    }
    if (!staged) {
        SHM_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s));
        return;
    }
    std::atomic<int> err{(int)cudaSuccess};
    host_tasks((int)((bytes + UPLOAD_SLOT - 1) / UPLOAD_SLOT), [&](int t) {
        const size_t at = (size_t)t * UPLOAD_SLOT, n = std::min(UPLOAD_SLOT, bytes - at);
        int i;
        {
            std::unique_lock<std::mutex> g(u->mu);
            u->cv.wait(g, [&] { return !u->idle.empty(); });  // one comes back when its thread has queued its copy
            i = u->idle.front();
            u->idle.pop_front();
        }
        cudaError_t e = cudaSetDevice(device);
        if (e == cudaSuccess) e = cudaEventSynchronize(u->ev[(size_t)i]);
        if (e == cudaSuccess) {
            uint8_t* p = u->pinned + (size_t)i * UPLOAD_SLOT;
            std::memcpy(p, (const uint8_t*)src + at, n);
            e = cudaMemcpyAsync((uint8_t*)dst + at, p, n, cudaMemcpyHostToDevice, s);
            if (e == cudaSuccess) e = cudaEventRecord(u->ev[(size_t)i], s);
        }
        if (e != cudaSuccess) err.store((int)e);
        {
            std::lock_guard<std::mutex> g(u->mu);
            u->idle.push_back(i);
        }
        u->cv.notify_one();
    });
    if (err.load() != (int)cudaSuccess) throw shm_cuda_error((cudaError_t)err.load());
}

}  // namespace shm
