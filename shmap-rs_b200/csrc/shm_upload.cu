// Host bytes in ordinary (pageable) memory on their way to the device. The
// driver's own copy from such memory goes through its staging buffers on the
// calling thread; here several threads fill a context's pinned slots, one each,
// and queue each slot's copy, so the bytes go up as fast as several cores read
// them. Bytes that are pinned already are copied from where they lie.
//
// The threads are the upload's own: on the packing threads it would hold up
// every context's host mapping, and wait for whole mapping calls itself. While
// a packing is in flight, in any context, they rest, and the driver's copy on
// the calling thread goes on by itself: the cores are the packing's.
//
// The copy takes this way from 64 MiB on, where both take the same time when
// the bytes are in the cores' caches (4.9 and 4.7 ms on 16 cores); for more
// bytes than those hold the threads are faster (240 MiB 24.7 and 11.0 ms), for
// fewer the driver is (16 MiB 1.1 and 1.7 ms: the threads have to start, and a
// slot's copy costs a call). Slots of 256 KiB took 17 ms for 256 MiB, of 1 MiB
// 12: the queueing calls of all threads take turns.
#include <algorithm>
#include <atomic>
#include <chrono>
#include <cstring>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>

#include "shm_internal.hpp"
#include "../host/pack.hpp"

namespace shm {

constexpr size_t UPLOAD_SLOT = (size_t)2 << 20;  // bytes
constexpr size_t UPLOAD_SLOTS = 8;               // 16 MiB a context, made when first needed; a thread each
constexpr size_t UPLOAD_LEAST = (size_t)64 << 20;

struct UploadStage {
    std::mutex use;  // one upload at a time
    uint8_t* pinned = nullptr;
    std::vector<cudaEvent_t> ev;  // slot's last copy
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
    std::atomic<size_t> next{0};  // bytes taken
    std::atomic<int> err{(int)cudaSuccess};
    // thread i: the next part through slot i, until all are taken or one failed
    auto work = [&](size_t i) {
        cudaError_t e = cudaSetDevice(device);
        uint8_t* const p = u->pinned + i * UPLOAD_SLOT;
        while (e == cudaSuccess && err.load() == (int)cudaSuccess && next.load() < bytes) {
            const bool rest = packing_now();
            if (rest && i) {
                std::this_thread::sleep_for(std::chrono::microseconds(200));
                continue;
            }
            const size_t take = rest ? UPLOAD_SLOT * UPLOAD_SLOTS : UPLOAD_SLOT, at = next.fetch_add(take);
            if (at >= bytes) break;
            const size_t n = std::min(take, bytes - at);
            if (rest) {  // (the caller's)
                e = cudaMemcpyAsync((uint8_t*)dst + at, (const uint8_t*)src + at, n, cudaMemcpyHostToDevice, s);
                continue;
            }
            if ((e = cudaEventSynchronize(u->ev[i])) != cudaSuccess) break;
            std::memcpy(p, (const uint8_t*)src + at, n);
            e = cudaMemcpyAsync((uint8_t*)dst + at, p, n, cudaMemcpyHostToDevice, s);
            const cudaError_t r = cudaEventRecord(u->ev[i], s);
            if (e == cudaSuccess) e = r;
        }
        if (e != cudaSuccess) err.store((int)e);
    };
    std::vector<std::thread> th;
    try {
        th.reserve(UPLOAD_SLOTS);
        const size_t most = std::max(1u, std::thread::hardware_concurrency());
        for (size_t i = 1; i < std::min(UPLOAD_SLOTS, most); i++) th.emplace_back(work, i);
    } catch (const std::system_error&) {  // no more threads: those there are do it
    } catch (const std::bad_alloc&) {
    }
    work(0);
    for (std::thread& t : th) t.join();
    if (err.load() != (int)cudaSuccess) throw shm_cuda_error((cudaError_t)err.load());
}

}  // namespace shm
