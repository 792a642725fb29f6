// svo_hostcopy.cpp -- device to pageable host memory through pinned slots.
//
// A copy to pageable memory is staged by the driver on one thread, 21 GB/s
// whatever its size.  Here up to kWorkers threads each stage spans of their own
// through two pinned slots, the next chunk's transfer running while the
// previous one is copied out: 20 MB of node records 700 us (1,030 by the
// driver), 748 MB of edges 20 ms (35), bound by the threads' copies and the
// link.  4 threads take 10% longer, chunks of 512 KiB 25% (more events and
// hand-overs per byte).  From 4 MiB on, where it begins to pay for the threads'
// start: 3.1 MB into memory in use 206-215 us staged and 183-202 by the driver,
// 4.0 MB 218-226 and 228-262, 5.2 MB 265-294 and 296-312.
#include "svo_hostcopy.h"

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <new>
#include <thread>
#include <vector>

namespace svo::host {

namespace {
constexpr int kWorkers = 8;
constexpr size_t kChunk = 1 << 20;  // a slot
constexpr size_t kSpan = 2 << 20;   // a huge page
}  // namespace

struct CopyPool {
    struct Worker {
        cudaStream_t stream = nullptr;
        cudaEvent_t done[2] = {};
        unsigned char *slot[2] = {};
    };
    int device = 0;
    std::mutex mu;  // held for the whole copy: one at a time, others take the driver's path
    bool tried = false;
    cudaEvent_t start = nullptr;
    std::vector<Worker> w;

    bool init() {
        if (tried) return !w.empty();
        const unsigned cores = std::thread::hardware_concurrency();
        const int n = std::max(1, std::min<int>(kWorkers, (int)cores / 2));
        w.reserve((size_t)n);  // (the only step here that throws: nothing is held yet)
        tried = true;
        bool ok = cudaEventCreateWithFlags(&start, cudaEventDisableTiming) == cudaSuccess;
        for (int i = 0; i < n && ok; ++i) {
            Worker k;
            ok = cudaStreamCreateWithFlags(&k.stream, cudaStreamNonBlocking) == cudaSuccess;
            for (int j = 0; j < 2 && ok; ++j)
                ok = cudaEventCreateWithFlags(&k.done[j], cudaEventDisableTiming) == cudaSuccess &&
                     cudaHostAlloc(reinterpret_cast<void **>(&k.slot[j]), kChunk, cudaHostAllocDefault) == cudaSuccess;
            w.push_back(k);
        }
        if (!ok) {
            cudaGetLastError();
            release();
        }
        return ok;
    }
    void release() {
        for (Worker &k : w) {
            for (int j = 0; j < 2; ++j) {
                if (k.done[j]) cudaEventDestroy(k.done[j]);
                if (k.slot[j]) cudaFreeHost(k.slot[j]);
            }
            if (k.stream) cudaStreamDestroy(k.stream);
        }
        w.clear();
        if (start) cudaEventDestroy(start);
        start = nullptr;
    }
    ~CopyPool() {
        if (w.empty()) return;
        cudaSetDevice(device);
        release();
    }
};

std::shared_ptr<CopyPool> copy_pool_create(int device) {
    auto p = std::make_shared<CopyPool>();
    p->device = device;
    return p;
}

bool copy_to_pageable(CopyPool &pool, void *dst, const void *src, size_t bytes, cudaStream_t st, cudaError_t *err) {
    if (bytes < 4 * kChunk) return false;
    std::unique_lock<std::mutex> lk(pool.mu, std::try_to_lock);
    if (!lk.owns_lock()) return false;
    std::vector<std::thread> threads;
    std::vector<size_t> here;  // the shares copied by this thread
    try {
        if (!pool.init()) return false;
        threads.reserve(pool.w.size());  // nothing below allocates beside a thread's start
        here.reserve(pool.w.size());
    } catch (const std::bad_alloc &) {
        return false;
    }
    if ((*err = cudaEventRecord(pool.start, st)) != cudaSuccess) return true;
    // The caller's capture mode holds for the threads that copy for it.
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    if ((*err = cudaThreadExchangeStreamCaptureMode(&mode)) != cudaSuccess) return true;
    cudaStreamCaptureMode relaxed = mode;
    cudaThreadExchangeStreamCaptureMode(&relaxed);
    // Spans end at multiples of kSpan in the destination's addresses, so that no
    // two threads fault the same huge page in.
    const size_t skew = (size_t)(reinterpret_cast<uintptr_t>(dst) % kSpan);
    const size_t spans = (bytes + skew + kSpan - 1) / kSpan;
    const size_t nw = std::min(pool.w.size(), spans);
    std::atomic<int> first_error{cudaSuccess};
    auto work = [&](size_t i) {
        CopyPool::Worker &k = pool.w[i];
        cudaStreamCaptureMode own = mode;
        cudaError_t e = cudaThreadExchangeStreamCaptureMode(&own);
        if (e == cudaSuccess) e = cudaSetDevice(pool.device);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(k.stream, pool.start, 0);
        size_t at[2] = {0, 0}, len[2] = {0, 0};  // what the slots hold (len 0: nothing)
        auto drain = [&](int j) {
            if (e == cudaSuccess && len[j]) e = cudaEventSynchronize(k.done[j]);
            if (e == cudaSuccess && len[j]) std::memcpy(static_cast<unsigned char *>(dst) + at[j], k.slot[j], len[j]);
            len[j] = 0;
        };
        int j = 0;
        for (size_t sp = i; sp < spans && e == cudaSuccess; sp += nw) {
            const size_t end = std::min(bytes, (sp + 1) * kSpan - skew);
            for (size_t c = sp ? sp * kSpan - skew : 0; c < end && e == cudaSuccess; c += len[j], j ^= 1) {
                drain(j);  // (empty after the other slot's turn below)
                if (e != cudaSuccess) break;
                at[j] = c;
                len[j] = std::min(kChunk, end - c);
                e = cudaMemcpyAsync(k.slot[j], static_cast<const unsigned char *>(src) + c, len[j], cudaMemcpyDeviceToHost,
                                    k.stream);
                if (e == cudaSuccess) e = cudaEventRecord(k.done[j], k.stream);
                drain(j ^ 1);
            }
        }
        drain(0);
        drain(1);
        if (e != cudaSuccess) {
            cudaStreamSynchronize(k.stream);  // nothing may still write to the slots
            int none = cudaSuccess;
            first_error.compare_exchange_strong(none, (int)e);
        }
    };
    here.push_back(0);
    for (size_t i = 1; i < nw; ++i) {
        try {
            threads.emplace_back(work, i);
        } catch (...) {  // no thread to be had: this share is copied here
            here.push_back(i);
        }
    }
    for (size_t i : here) work(i);
    for (std::thread &t : threads) t.join();
    *err = (cudaError_t)first_error.load();
    return true;
}

}  // namespace svo::host
