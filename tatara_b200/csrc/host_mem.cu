// The pool of page-locked blocks and the copying helper threads.
//
// Page-locking is what a loader's batch costs when every batch allocates its arrays: cudaHostAlloc and cudaFreeHost pin and
// unpin page by page and wait for the device (18 ms for the six arrays of 65 536 positions; the extraction itself moves 24 MB).
// Freed blocks are therefore kept, up to POOL_LIMIT bytes in all, and handed out again for requests of the same size class.
// A block that no request has matched for POOL_AGE allocations goes back to the system, as does everything when an
// allocation fails.
//
// cudaFreeHost waits for the device, so work that still reads or writes a freed block is safe with it, whoever queued it and
// on whichever stream.  The pool keeps that: before blocks freed since the last allocation are handed out again, one event per
// GPU captures all work queued there (cuCtxRecordEvent), and a block goes out only behind them.  The events are recorded in
// the contexts this process has open, whichever device is current: the thread that drops a batch need not be on the GPU that
// reads it, and freeing makes no CUDA call.  (An event at every free instead: 4 us each, 5 % of the extraction of 65 536
// records into page-locked arrays.)
#include "host_mem.cuh"

#include <cuda.h>
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

// the driver's functions, without a link-time dependency on it
struct Driver {
    CUresult (*DeviceGetCount)(int*) = nullptr;
    CUresult (*DeviceGet)(CUdevice*, int) = nullptr;
    CUresult (*PrimaryCtxGetState)(CUdevice, unsigned*, int*) = nullptr;
    CUresult (*PrimaryCtxRetain)(CUcontext*, CUdevice) = nullptr;
    CUresult (*PrimaryCtxRelease)(CUdevice) = nullptr;
    CUresult (*CtxPushCurrent)(CUcontext) = nullptr;
    CUresult (*CtxPopCurrent)(CUcontext*) = nullptr;
    CUresult (*CtxRecordEvent)(CUcontext, CUevent) = nullptr;
    CUresult (*EventCreate)(CUevent*, unsigned) = nullptr;
    CUresult (*EventQuery)(CUevent) = nullptr;
    CUresult (*EventSynchronize)(CUevent) = nullptr;
    bool ok = true;
    Driver() {
        auto get = [&](const char* name, void* fn) {
            cudaDriverEntryPointQueryResult r;
            if (cudaGetDriverEntryPointByVersion(name, (void**)fn, 12050, cudaEnableDefault, &r) != cudaSuccess || r != cudaDriverEntryPointSuccess || !*(void**)fn) {
                cudaGetLastError();
                ok = false;
            }
        };
        get("cuDeviceGetCount", &DeviceGetCount); get("cuDeviceGet", &DeviceGet);
        get("cuDevicePrimaryCtxGetState", &PrimaryCtxGetState); get("cuDevicePrimaryCtxRetain", &PrimaryCtxRetain);
        get("cuDevicePrimaryCtxRelease", &PrimaryCtxRelease); get("cuCtxPushCurrent", &CtxPushCurrent); get("cuCtxPopCurrent", &CtxPopCurrent);
        get("cuCtxRecordEvent", &CtxRecordEvent); get("cuEventCreate", &EventCreate); get("cuEventQuery", &EventQuery);
        get("cuEventSynchronize", &EventSynchronize);
    }
};
Driver& driver() { static Driver* d = new Driver; return *d; }

struct Guard { int dev; CUevent ev; };  // work queued on a GPU

typedef std::vector<Guard> Guards;
const size_t POOL_BUSY = 2;  // blocks of a size class that may be waited for; with fewer a new one is allocated

struct Block {
    void* p;
    size_t size;
    uint64_t freed_at;
    std::shared_ptr<Guards> guards;  // shared by the blocks freed between two allocations; none yet: freed since the last one
};

struct Pool {
    std::mutex mu;
    std::unordered_map<void*, size_t> live;
    std::vector<Block> cached;  // oldest first
    std::vector<Guard> spare;   // events to record again
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

// (the callers hold the pool's mutex)
// false: some GPU's work could not be captured (a driver without the call, a stream being captured)
bool record_guards(Pool& P, Guards& out) {
    Driver& D = driver();
    int n = 0;
    if (!D.ok || D.DeviceGetCount(&n) != CUDA_SUCCESS) return false;
    bool all = true;
    for (int i = 0; i < n; ++i) {
        CUdevice dev;
        unsigned flags;
        int active = 0;
        if (D.DeviceGet(&dev, i) != CUDA_SUCCESS || D.PrimaryCtxGetState(dev, &flags, &active) != CUDA_SUCCESS) { all = false; continue; }
        if (!active) continue;
        CUcontext ctx, popped;
        if (D.PrimaryCtxRetain(&ctx, dev) != CUDA_SUCCESS) { all = false; continue; }
        if (D.CtxPushCurrent(ctx) == CUDA_SUCCESS) {
            Guard g{i, nullptr};
            for (size_t k = 0; k < P.spare.size(); ++k)
                if (P.spare[k].dev == i) { g = P.spare[k]; P.spare.erase(P.spare.begin() + k); break; }
            if (g.ev || D.EventCreate(&g.ev, CU_EVENT_DISABLE_TIMING) == CUDA_SUCCESS) {
                if (D.CtxRecordEvent(ctx, g.ev) == CUDA_SUCCESS) out.push_back(g);
                else { all = false; P.spare.push_back(g); }
            } else all = false;
            D.CtxPopCurrent(&popped);
        } else all = false;
        D.PrimaryCtxRelease(dev);
    }
    return all;
}

void guard_new_blocks(Pool& P) {
    std::shared_ptr<Guards> g;
    for (Block& b : P.cached) {
        if (b.guards) continue;
        if (!g) {
            g = std::make_shared<Guards>();
            if (!record_guards(P, *g)) { P.spare.insert(P.spare.end(), g->begin(), g->end()); return; }
        }
        b.guards = g;
    }
}

// Work that is known to be done needs no events: they are recorded again for later blocks (a query costs 1 us, a wait 2).
void drop_guards(Pool& P, Guards& g) {
    P.spare.insert(P.spare.end(), g.begin(), g.end());
    g.clear();
}

bool idle(Pool& P, const Block& b) {
    for (const Guard& g : *b.guards)
        if (driver().EventQuery(g.ev) == CUDA_ERROR_NOT_READY) return false;
    drop_guards(P, *b.guards);
    return true;
}

// Not under the mutex: a copy of the events, which another thread may meanwhile find done and record again.  The wait then is
// for later work as well, never for less.
void wait_guards(const Guards& guards) {
    for (const Guard& g : guards) driver().EventSynchronize(g.ev);
}

void release(std::vector<Block>& out) {
    for (Block& b : out) cudaFreeHost(b.p);  // waits by itself
    out.clear();
}

}  // namespace

void* pinned_alloc(size_t bytes) {
    Pool& P = pool();
    const size_t size = size_class(bytes);
    std::vector<Block> old;
    Block hit{nullptr, 0, 0, nullptr};
    Guards events;  // to wait for
    {
        std::lock_guard<std::mutex> lock(P.mu);
        ++P.tick;
        guard_new_blocks(P);
        // the most recently freed block that nothing uses any more (its pages are the likeliest to be in a cache); else the
        // one that was freed first, once there are so many that the next call finds an idle one
        size_t at = P.cached.size(), busy = 0;
        bool found = false;
        const Guards* running = nullptr;
        for (size_t i = P.cached.size(); i-- > 0 && !found;)
            if (P.cached[i].size == size && P.cached[i].guards) {
                at = i;
                found = P.cached[i].guards.get() != running && idle(P, P.cached[i]);
                if (!found) { running = P.cached[i].guards.get(); ++busy; }
            }
        if (found || busy >= POOL_BUSY) {
            if (!found) events = *P.cached[at].guards;
            hit = std::move(P.cached[at]);
            P.cached.erase(P.cached.begin() + at);
            P.cached_bytes -= size;
            P.live[hit.p] = size;
        }
        while (!P.cached.empty() && P.cached.front().freed_at + POOL_AGE < P.tick) {
            P.cached_bytes -= P.cached.front().size;
            old.push_back(std::move(P.cached.front()));
            P.cached.erase(P.cached.begin());
        }
    }
    release(old);
    if (hit.p) {
        wait_guards(events);
        if (!events.empty()) {
            std::lock_guard<std::mutex> lock(P.mu);
            drop_guards(P, *hit.guards);
        }
        return hit.p;
    }
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
        P.cached.push_back({p, it->second, P.tick, nullptr});
        P.cached_bytes += it->second;
        P.live.erase(it);
        while (P.cached_bytes > POOL_LIMIT) {
            P.cached_bytes -= P.cached.front().size;
            out.push_back(std::move(P.cached.front()));
            P.cached.erase(P.cached.begin());
        }
    }
    release(out);
    return true;
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
