// The pool of page-locked blocks and the copying helper threads.
//
// Page-locking is what a loader's batch costs when every batch allocates its arrays: cudaHostAlloc and cudaFreeHost pin and
// unpin page by page and wait for the device (18 ms for the six arrays of 65 536 positions; the extraction itself moves 24 MB).
// Freed blocks are therefore kept, up to POOL_LIMIT bytes in all, and handed out again for requests of the same size class.
// A block that no request has matched for POOL_AGE allocations goes back to the system, as does everything when an
// allocation fails.
#include "host_mem.cuh"

#include <stdint.h>
#include <string.h>
#ifdef __SSE2__
#include <emmintrin.h>
#endif

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <memory>
#include <mutex>
#include <thread>
#include <unordered_map>
#include <vector>

namespace {

const size_t POOL_LIMIT = (size_t)256 << 20;  // five full batches of index arrays
const uint64_t POOL_AGE = 256;

struct Block {
    void* p;
    size_t size;
    uint64_t freed_at;
    std::vector<cudaEvent_t> events;  // copies that may still read the block
};

struct Pool {
    std::mutex mu;
    std::unordered_map<void*, size_t> live;
    std::vector<Block> cached;  // oldest first
    std::vector<cudaStream_t> watched;
    size_t cached_bytes = 0;
    uint64_t tick = 0;
};
// never destroyed: blocks may be given back after static destructors have begun, and the driver releases what is left
Pool& pool() { static Pool* p = new Pool; return *p; }

// size classes: sixteen steps per power of two, so that at most 1/16 of a block is unused
size_t size_class(size_t n) {
    if (n < 4096) return 4096;
    size_t step = 4096;
    while (step * 32 <= n) step *= 2;
    return (n + step - 1) / step * step;
}

void wait_events(Block& b) {
    for (cudaEvent_t e : b.events) { cudaEventSynchronize(e); cudaEventDestroy(e); }
    b.events.clear();
}

void release(std::vector<Block>& out) {
    for (Block& b : out) { wait_events(b); cudaFreeHost(b.p); }
    out.clear();
}

}  // namespace

void* pinned_alloc(size_t bytes) {
    Pool& P = pool();
    const size_t size = size_class(bytes);
    std::vector<Block> old;
    Block hit{nullptr, 0, 0, {}};
    {
        std::lock_guard<std::mutex> lock(P.mu);
        ++P.tick;
        for (size_t i = P.cached.size(); i-- > 0;)
            if (P.cached[i].size == size) {  // the most recently used one: its pages are the likeliest to be in a cache
                hit = std::move(P.cached[i]);
                P.cached.erase(P.cached.begin() + i);
                P.cached_bytes -= size;
                P.live[hit.p] = size;
                break;
            }
        while (!P.cached.empty() && P.cached.front().freed_at + POOL_AGE < P.tick) {
            P.cached_bytes -= P.cached.front().size;
            old.push_back(std::move(P.cached.front()));
            P.cached.erase(P.cached.begin());
        }
    }
    release(old);
    if (hit.p) { wait_events(hit); return hit.p; }
    void* p = nullptr;
    if (cudaHostAlloc(&p, size, cudaHostAllocDefault) != cudaSuccess) {
        cudaGetLastError();
        pinned_trim();
        if (cudaHostAlloc(&p, size, cudaHostAllocDefault) != cudaSuccess) { cudaGetLastError(); return nullptr; }
    }
    std::lock_guard<std::mutex> lock(P.mu);
    P.live[p] = size;
    return p;
}

bool pinned_free(void* p) {
    Pool& P = pool();
    std::vector<Block> out;
    {
        std::lock_guard<std::mutex> lock(P.mu);
        auto it = P.live.find(p);
        if (it == P.live.end()) return false;
        Block b{p, it->second, P.tick, {}};
        P.live.erase(it);
        for (cudaStream_t s : P.watched) {
            cudaEvent_t e;
            if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) { cudaGetLastError(); continue; }
            if (cudaEventRecord(e, s) == cudaSuccess) b.events.push_back(e);
            else { cudaGetLastError(); cudaEventDestroy(e); }
        }
        P.cached_bytes += b.size;
        P.cached.push_back(std::move(b));
        while (P.cached_bytes > POOL_LIMIT) {
            P.cached_bytes -= P.cached.front().size;
            out.push_back(std::move(P.cached.front()));
            P.cached.erase(P.cached.begin());
        }
    }
    release(out);
    return true;
}

void pinned_watch_stream(cudaStream_t s) {
    std::lock_guard<std::mutex> lock(pool().mu);
    pool().watched.push_back(s);
}

void pinned_unwatch_stream(cudaStream_t s) {
    std::lock_guard<std::mutex> lock(pool().mu);
    auto& w = pool().watched;
    w.erase(std::remove(w.begin(), w.end(), s), w.end());
}

void pinned_trim() {
    std::vector<Block> out;
    {
        std::lock_guard<std::mutex> lock(pool().mu);
        out.swap(pool().cached);
        pool().cached_bytes = 0;
    }
    release(out);
}

// ---- helper threads --------------------------------------------------------------------------------------------------
// A job is a range of indices handed out by an atomic counter.  The caller takes indices like any helper and waits only for
// indices that a helper has already taken, so a job ends also where no helper exists (one core, or a forked child).
namespace {

struct Job {
    const std::function<void(int)>* work;
    int n;
    std::atomic<int> next{0};
    std::unique_ptr<std::atomic<char>[]> done;
};

struct Helpers {
    std::mutex mu;
    std::condition_variable wake;
    std::vector<std::shared_ptr<Job>> jobs;  // jobs with indices left
    int threads = 0;

    void run() {
        for (;;) {
            std::shared_ptr<Job> j;
            {
                std::unique_lock<std::mutex> lock(mu);
                wake.wait(lock, [&] { return !jobs.empty(); });
                j = jobs.front();
            }
            for (int i; (i = j->next.fetch_add(1)) < j->n;) {
                (*j->work)(i);
                j->done[i].store(1, std::memory_order_release);
            }
            std::lock_guard<std::mutex> lock(mu);
            jobs.erase(std::remove(jobs.begin(), jobs.end(), j), jobs.end());
        }
    }
    Helpers() {
        // a memcpy stream per core saturates the memory at about eight; the caller is one of them
        const int cores = (int)std::thread::hardware_concurrency();
        const int want = std::max(0, std::min(7, cores - 1));
        for (int i = 0; i < want; ++i) {
            try { std::thread([this] { run(); }).detach(); ++threads; } catch (...) { break; }
        }
    }
};
Helpers& helpers() { static Helpers* h = new Helpers; return *h; }  // lives as long as the process, like its threads

const size_t COPY_PIECE = (size_t)256 << 10;

}  // namespace

void host_parallel(int n, const std::function<void(int)>& work, const std::function<void(int)>& in_order) {
    if (n <= 1) {
        if (n == 1) { work(0); if (in_order) in_order(0); }
        return;
    }
    Helpers& H = helpers();
    auto j = std::make_shared<Job>();
    j->work = &work;
    j->n = n;
    j->done.reset(new std::atomic<char>[n]);
    for (int i = 0; i < n; ++i) j->done[i].store(0, std::memory_order_relaxed);
    if (H.threads > 0) {
        { std::lock_guard<std::mutex> lock(H.mu); H.jobs.push_back(j); }
        H.wake.notify_all();
    }
    int sent = 0;
    auto send = [&] {
        while (sent < n && j->done[sent].load(std::memory_order_acquire)) { if (in_order) in_order(sent); ++sent; }
    };
    for (int i; (i = j->next.fetch_add(1)) < n;) {
        work(i);
        j->done[i].store(1, std::memory_order_release);
        send();
    }
    if (H.threads > 0) {
        std::lock_guard<std::mutex> lock(H.mu);
        H.jobs.erase(std::remove(H.jobs.begin(), H.jobs.end(), j), H.jobs.end());
    }
    while (sent < n) { send(); if (sent < n) std::this_thread::yield(); }
}

void host_copy_for_device(void* dst, const void* src, size_t bytes) {
#ifdef __SSE2__
    char* d = static_cast<char*>(dst);
    const char* s = static_cast<const char*>(src);
    const size_t head = std::min(bytes, (size_t)(-(intptr_t)d & 15));
    memcpy(d, s, head);
    size_t i = head;
    for (; i + 64 <= bytes; i += 64) {
        _mm_prefetch(s + i + 1024, _MM_HINT_NTA);  // past the end of the source a prefetch is dropped
        const __m128i a = _mm_loadu_si128((const __m128i*)(s + i)), b = _mm_loadu_si128((const __m128i*)(s + i + 16));
        const __m128i c = _mm_loadu_si128((const __m128i*)(s + i + 32)), e = _mm_loadu_si128((const __m128i*)(s + i + 48));
        _mm_stream_si128((__m128i*)(d + i), a);
        _mm_stream_si128((__m128i*)(d + i + 16), b);
        _mm_stream_si128((__m128i*)(d + i + 32), c);
        _mm_stream_si128((__m128i*)(d + i + 48), e);
    }
    memcpy(d + i, s + i, bytes - i);
    _mm_sfence();
#else
    memcpy(dst, src, bytes);
#endif
}

void host_stage(void* dst, const void* src, size_t bytes) {
    const int n = (int)((bytes + COPY_PIECE - 1) / COPY_PIECE);
    if (n < 4) { host_copy_for_device(dst, src, bytes); return; }  // below 1 MB waking a thread costs more than it saves
    host_parallel(n, [&](int i) {
        const size_t o = (size_t)i * COPY_PIECE;
        host_copy_for_device((char*)dst + o, (const char*)src + o, std::min(COPY_PIECE, bytes - o));
    });
}

void host_copy_out(const HostCopy* items, int n) {
    // Pieces end on 2 MB boundaries of the destination: it is often fresh memory, and two threads that touch the same huge
    // page for the first time would both clear it.
    const size_t page = (size_t)2 << 20;
    std::vector<HostCopy> pieces;
    size_t total = 0;
    for (int k = 0; k < n; ++k) {
        total += items[k].bytes;
        for (size_t o = 0; o < items[k].bytes;) {
            const size_t to_edge = page - ((uintptr_t)items[k].dst + o) % page, b = std::min(to_edge, items[k].bytes - o);
            pieces.push_back({(char*)items[k].dst + o, (const char*)items[k].src + o, b});
            o += b;
        }
    }
    auto copy = [&](int i) { memcpy(pieces[i].dst, pieces[i].src, pieces[i].bytes); };
    if (total < 4 * COPY_PIECE) for (int i = 0; i < (int)pieces.size(); ++i) copy(i);
    else host_parallel((int)pieces.size(), copy);
}
