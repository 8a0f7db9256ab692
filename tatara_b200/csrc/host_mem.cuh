// Host-side memory of the library: the pool of page-locked blocks behind tb_host_alloc and the helper threads that copy
// pageable arrays (host_mem.cu).
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

#include <functional>

// Runs work(0) .. work(n - 1) on the calling thread and the library's helper threads.  in_order(i), when given, runs on the
// calling thread for ascending i, each as soon as work(0 .. i) are done: an upload sends a piece off while later ones are
// still being copied.  Several threads may call at once.
void host_parallel(int n, const std::function<void(int)>& work, const std::function<void(int)>& in_order = nullptr);

// memcpy into memory that the device reads next (on the calling thread): stores past the caches.  Lines that are dirty in the caches of several cores
// slow the device's reads down to a third (22 MB just written by eight threads: 1.0 ms against 0.43 ms).
void host_copy_for_device(void* dst, const void* src, size_t bytes);
// the same, shared among the helper threads when it is large enough to pay
void host_stage(void* dst, const void* src, size_t bytes);
struct HostCopy { void* dst; const void* src; size_t bytes; };
// memcpy of n arrays to the caller's memory, shared among the helper threads when it is large enough to pay
void host_copy_out(const HostCopy* items, int n);

// page-locked memory from the pool; NULL when none can be had
void* pinned_alloc(size_t bytes);
// false: not a block of the pool.  The block is not handed out again before the work that any GPU has queued by then is done.
bool pinned_free(void* p);
// frees every cached block (called when memory runs out)
void pinned_trim();
