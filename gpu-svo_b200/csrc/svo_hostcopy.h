// svo_hostcopy.h -- staged copies from device memory to pageable host memory.
#pragma once
#include <cstddef>
#include <memory>

#include <cuda_runtime.h>

namespace svo::host {

// Pinned slots, streams and events for staged copies (16 MiB at most, made by
// the first copy that needs them).  A context and its results share one; the
// last of them frees it.
struct CopyPool;
std::shared_ptr<CopyPool> copy_pool_create(int device);

// Copies `bytes` from device memory, as the work on `st` before leaves it, to
// pageable host memory and waits for it; *err is the outcome.  False: not done
// (a small copy, another thread's copy in progress, no pinned memory): copy
// some other way.
bool copy_to_pageable(CopyPool &pool, void *dst, const void *src, size_t bytes, cudaStream_t st, cudaError_t *err);

}  // namespace svo::host
