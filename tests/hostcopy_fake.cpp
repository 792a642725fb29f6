// Drives svo::host::copy_to_pageable on the CPU against a stand-in for the CUDA
// runtime (device memory is host memory, copies are memcpy), with failures made
// on the host: an allocation, a thread or a copy that fails.  Built by
// test_hostcopy_faults.py together with svo_hostcopy.cpp; every check that does
// not hold is printed and counted in the exit code.
#include <atomic>
#include <cerrno>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <new>
#include <thread>
#include <vector>

#include <dlfcn.h>
#include <pthread.h>

#include "svo_hostcopy.h"

namespace {
std::atomic<long> g_new_left{-1};     // allocations until one fails (-1: never)
std::atomic<long> g_thread_left{-1};  // threads until none can be made any more
std::atomic<long> g_copy_left{-1};    // copies until one fails
std::atomic<long> g_alive{0};         // runtime objects not given back

bool count_down(std::atomic<long> &n, bool once) {
    long k = n.load();
    while (k >= 0 && !n.compare_exchange_weak(k, k == 0 ? (once ? -1 : 0) : k - 1)) {
    }
    return k == 0;
}
}  // namespace

void *operator new(std::size_t n) {
    if (count_down(g_new_left, true)) throw std::bad_alloc();
    if (void *p = std::malloc(n ? n : 1)) return p;
    throw std::bad_alloc();
}
void operator delete(void *p) noexcept { std::free(p); }
void operator delete(void *p, std::size_t) noexcept { std::free(p); }

extern "C" {
int pthread_create(pthread_t *t, const pthread_attr_t *a, void *(*f)(void *), void *arg) {
    using Fn = int (*)(pthread_t *, const pthread_attr_t *, void *(*)(void *), void *);
    static Fn real = reinterpret_cast<Fn>(dlsym(RTLD_NEXT, "pthread_create"));
    if (count_down(g_thread_left, false)) return EAGAIN;
    return real(t, a, f, arg);
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) {
    *e = reinterpret_cast<cudaEvent_t>(std::malloc(1));
    ++g_alive;
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) {
    std::free(e);
    --g_alive;
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
    *s = reinterpret_cast<cudaStream_t>(std::malloc(1));
    ++g_alive;
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
    std::free(s);
    --g_alive;
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) {
    *p = std::malloc(n);
    ++g_alive;
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) {
    std::free(p);
    --g_alive;
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
    if (count_down(g_copy_left, true)) return cudaErrorInvalidValue;
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode *) { return cudaSuccess; }
}

namespace {
int g_bad = 0;
void expect(bool ok, const char *what, long k) {
    if (ok) return;
    ++g_bad;
    std::printf("%s (%ld)\n", what, k);
}

constexpr size_t kBytes = (37u << 20) + 12345;

// One copy into a cleared destination at an odd offset, by a pool of its own or `pool`.
void one_copy(std::shared_ptr<svo::host::CopyPool> pool, std::atomic<long> *fault, long k, bool may_fail) {
    static std::vector<unsigned char> src, dst(kBytes + 64);
    if (src.empty()) {
        src.resize(kBytes);
        for (size_t i = 0; i < kBytes; ++i) src[i] = (unsigned char)(i * 2654435761u >> 13);
    }
    std::memset(dst.data(), 0, dst.size());
    cudaError_t err = cudaSuccess;
    bool done = false;
    if (fault) fault->store(k);
    try {
        done = svo::host::copy_to_pageable(*pool, dst.data() + 7, src.data(), kBytes, nullptr, &err);
    } catch (...) {
        expect(false, "an exception left the copy", k);
    }
    if (fault) fault->store(-1);
    if (done && err == cudaSuccess) expect(std::memcmp(dst.data() + 7, src.data(), kBytes) == 0, "wrong bytes", k);
    else expect(may_fail, "the copy was not made", k);
}
}  // namespace

int main() {
    {
        auto pool = svo::host::copy_pool_create(0);
        one_copy(pool, nullptr, 0, false);
        for (long k = 0; k < 8; ++k) one_copy(pool, &g_thread_left, k, false);  // no thread: the shares are copied here
        for (long k = 0; k < 40; k += 3) one_copy(pool, &g_copy_left, k, true);
        for (long k = 0; k < 40; ++k) one_copy(pool, &g_new_left, k, true);
        one_copy(pool, nullptr, 0, false);  // and the pool still works
    }
    for (long k = 0; k < 40; ++k) {  // the first copy of a pool
        auto pool = svo::host::copy_pool_create(0);
        one_copy(pool, &g_new_left, k, true);
        one_copy(pool, nullptr, k, false);
    }
    for (long k = 0; k < 3; ++k) {  // no memory and no thread at once
        auto pool = svo::host::copy_pool_create(0);
        one_copy(pool, nullptr, 0, false);
        g_thread_left.store(2);
        one_copy(pool, &g_new_left, 2 + k, true);
        g_thread_left.store(-1);
    }
    expect(g_alive.load() == 0, "runtime objects left", g_alive.load());
    std::printf("%d bad\n", g_bad);
    return g_bad ? 1 : 0;
}
