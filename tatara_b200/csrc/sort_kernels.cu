// Small-key stable counting sorts over many blocks (keys < 128):
//  - positions by LayerStack bucket  -> `order`, bucket segments, dense tiles and work units
//    (replaces count_buckets / exclusive_scan_aligned / scatter_bucket_perm, native_kernels.cu:1858-1925)
//  - (position, perspective) items by the king bucket of their feature rows -> `items`, so that blocks that
//    run at the same time gather from the same slice of the FT table and the slice stays in L2.
// Both sorts share three launches (blockIdx.y / blockIdx.x selects the sort): per-block histogram, one-block scan of the
// [key][block] matrix, stable scatter (rank inside a block = warp match + prefix over the block's warps); a fourth
// launch cuts the segments into what the later kernels work on.  Results do not depend on timing.
#include "common.cuh"
#include "ft_slice.cuh"

#define SORT_BLOCK 1024
#define SORT_MAX_KEYS 128

struct BucketKey {
    const int* bucket;  // may be NULL: one group
    int nb;
    __device__ int operator()(int i) const {
        const int k = bucket ? bucket[i] : 0;
        return (unsigned)k < (unsigned)nb ? k : nb;  // out-of-range ids form the last group
    }
};

// item i < B is the stm perspective of position i, item B + b the nstm perspective of position b.  The key is
// the table slice (index / rows_per_slice) of the item's first feature; items without one go last.
struct ItemKey {
    const int* idx_stm;
    const int* idx_nstm;
    const int* nnz;
    int B, A, N, rows_per_slice, n_slices;
    __device__ int operator()(int i) const {
        const int p = i >= B, b = i - p * B;
        if (nnz[b] <= 0) return n_slices;
        const int f = (p ? idx_nstm : idx_stm)[(size_t)b * A];
        return (unsigned)f < (unsigned)N ? f / rows_per_slice : n_slices;
    }
};

template <class KeyFn>
static __device__ __forceinline__ void sort_hist_body(KeyFn fn, int n, int K, int G, int* __restrict__ hist, int* s_h, int block) {
    if (threadIdx.x < SORT_MAX_KEYS) s_h[threadIdx.x] = 0;
    __syncthreads();
    const int i = block * SORT_BLOCK + threadIdx.x;
    if (i < n) atomicAdd(&s_h[fn(i)], 1);
    __syncthreads();
    if ((int)threadIdx.x < K) hist[threadIdx.x * G + block] = s_h[threadIdx.x];
}

// two independent sorts in one launch: blockIdx.y selects the sort
template <class Fn0, class Fn1>
__global__ void __launch_bounds__(SORT_BLOCK) k_sort_hist2(Fn0 f0, int n0, int K0, int G0, int* __restrict__ h0, Fn1 f1, int n1, int K1,
                                                            int G1, int* __restrict__ h1) {
    __shared__ int s_h[SORT_MAX_KEYS];
    if (blockIdx.y == 0) { if ((int)blockIdx.x < G0) sort_hist_body(f0, n0, K0, G0, h0, s_h, blockIdx.x); }
    else if ((int)blockIdx.x < G1) sort_hist_body(f1, n1, K1, G1, h1, s_h, blockIdx.x);
}

// exclusive scan of hist[K][G] in key-major order (in place); seg_start[k] = first output slot of key k
static __device__ __forceinline__ void sort_scan_body(int* __restrict__ hist, int K, int G, int n, int* __restrict__ seg_start, int* s_warp) {
    const int total = K * G;
    const int per = (total + 1023) / 1024;
    const int beg = min((int)threadIdx.x * per, total), end = min(beg + per, total);
    int sum = 0;
    for (int i = beg; i < end; ++i) sum += hist[i];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int incl = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += t;
    }
    if (lane == 31) s_warp[w] = incl;
    __syncthreads();
    if (w == 0) {
        const int t = s_warp[lane];
        int ti = t;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, ti, d);
            if (lane >= d) ti += u;
        }
        s_warp[lane] = ti - t;
    }
    __syncthreads();
    int run = s_warp[w] + incl - sum;
    for (int i = beg; i < end; ++i) {
        const int c = hist[i];
        hist[i] = run;
        if (i % G == 0) seg_start[i / G] = run;
        run += c;
    }
    if (threadIdx.x == 0) seg_start[K] = n;
}

__global__ void __launch_bounds__(1024) k_sort_scan2(int* __restrict__ h0, int K0, int G0, int n0, int* __restrict__ seg0,
                                                      int* __restrict__ h1, int K1, int G1, int n1, int* __restrict__ seg1) {
    __shared__ int s_warp[32];
    if (blockIdx.x == 0) sort_scan_body(h0, K0, G0, n0, seg0, s_warp);
    else sort_scan_body(h1, K1, G1, n1, seg1, s_warp);
}

template <class KeyFn>
static __device__ __forceinline__ void sort_scatter_body(KeyFn fn, int n, int K, int G, const int* __restrict__ base, int* __restrict__ out,
                                                         int (*s_cnt)[SORT_MAX_KEYS], int block) {
    for (int e = threadIdx.x; e < 32 * SORT_MAX_KEYS; e += SORT_BLOCK) (&s_cnt[0][0])[e] = 0;
    __syncthreads();
    const int i = block * SORT_BLOCK + threadIdx.x;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int key = i < n ? fn(i) : -1;
    const unsigned peers = __match_any_sync(0xffffffffu, key);
    const int rank = __popc(peers & ((1u << lane) - 1u));
    if (rank == 0 && key >= 0) s_cnt[w][key] = __popc(peers);
    __syncthreads();
    if ((int)threadIdx.x < K) {
        int run = 0;
        for (int ww = 0; ww < 32; ++ww) {
            const int c = s_cnt[ww][threadIdx.x];
            s_cnt[ww][threadIdx.x] = run;
            run += c;
        }
    }
    __syncthreads();
    if (key >= 0) out[base[key * G + block] + s_cnt[w][key] + rank] = i;
}

template <class Fn0, class Fn1>
__global__ void __launch_bounds__(SORT_BLOCK) k_sort_scatter2(Fn0 f0, int n0, int K0, int G0, const int* __restrict__ b0, int* __restrict__ o0,
                                                              Fn1 f1, int n1, int K1, int G1, const int* __restrict__ b1, int* __restrict__ o1) {
    __shared__ int s_cnt[32][SORT_MAX_KEYS];
    if (blockIdx.y == 0) { if ((int)blockIdx.x < G0) sort_scatter_body(f0, n0, K0, G0, b0, o0, s_cnt, blockIdx.x); }
    else if ((int)blockIdx.x < G1) sort_scatter_body(f1, n1, K1, G1, b1, o1, s_cnt, blockIdx.x);
}

// ---- what the kernels behind the sorts work on, one block each -------------------------------------------------------
// At most 128 keys; what depends on all of them is summed by a warp per key.  (One thread walking the keys took 14 us of
// a step for the forward runs and 17 us for the chunks.)
#define PLAN_THREADS 1024

// tiles: runs of <= TB_TILE_M positions of one bucket; units: runs of <= ut tiles of one bucket; weight units: of <= TB_UNIT_TILES
static __device__ void plan_tiles(const int* __restrict__ s_seg, int K, int ut, TileDesc* __restrict__ tiles, int* __restrict__ n_tiles,
                                  TileDesc* __restrict__ units, TileDesc* __restrict__ wunits) {
    __shared__ int s_tile_base[TB_MAX_BUCKETS + 3], s_unit_base[TB_MAX_BUCKETS + 3], s_wunit_base[TB_MAX_BUCKETS + 3];
    if (threadIdx.x == 0) {
        int trun = 0, urun = 0, wrun = 0;
        for (int k = 0; k <= K; ++k) {
            s_tile_base[k] = trun;
            s_unit_base[k] = urun;
            s_wunit_base[k] = n_tiles[3 + k] = wrun;
            if (k == K) break;
            const int nt = (s_seg[k + 1] - s_seg[k] + TB_TILE_M - 1) / TB_TILE_M;
            trun += nt;
            urun += (nt + ut - 1) / ut;
            wrun += (nt + TB_UNIT_TILES - 1) / TB_UNIT_TILES;
        }
        n_tiles[0] = trun;
        n_tiles[1] = urun;
        n_tiles[2] = wrun;
    }
    __syncthreads();
    for (int t = threadIdx.x; t < s_tile_base[K]; t += PLAN_THREADS) {
        int k = 0;
        while (s_tile_base[k + 1] <= t) ++k;
        const int i = t - s_tile_base[k];
        TileDesc d;
        d.start = s_seg[k] + i * TB_TILE_M;
        d.count = min(TB_TILE_M, s_seg[k + 1] - d.start);
        d.bucket = k;
        d.pad = 0;
        tiles[t] = d;
    }
    auto cut = [&](const int* base, int size, TileDesc* out) {
        for (int u = threadIdx.x; u < base[K]; u += PLAN_THREADS) {
            int k = 0;
            while (base[k + 1] <= u) ++k;
            TileDesc d;
            d.start = s_tile_base[k] + (u - base[k]) * size;
            d.count = min(size, s_tile_base[k + 1] - d.start);
            d.bucket = k;
            d.pad = 0;
            out[u] = d;
        }
    };
    cut(s_unit_base, ut, units);
    cut(s_wunit_base, TB_UNIT_TILES, wunits);
}

// Runs of the slice-resident forward: <= SLICE_IPC consecutive slots of one slice, the largest first.  The blocks take
// (run, column strip) units in this order: king-bucket slices differ in size by two and more (a mirrored board has a centre
// file), and with the units in slice order the busiest SM of a full batch worked 14 % longer than the average one.
static __device__ void plan_forward(const int* __restrict__ s_seg, int n_keys, FwdWork* __restrict__ work, int* __restrict__ n_work) {
    __shared__ int s_size[SORT_MAX_KEYS], s_n[SORT_MAX_KEYS];
    const int k = threadIdx.x;
    if (k < n_keys) {
        const int len = s_seg[k + 1] - s_seg[k];
        const int n = (len + SLICE_IPC - 1) / SLICE_IPC;
        s_n[k] = n;
        s_size[k] = n > 0 ? ((len + n - 1) / n + 127) & ~127 : 0;  // equal runs of whole rounds of 128 items
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    for (int key = threadIdx.x >> 5; key < n_keys; key += PLAN_THREADS / 32) {
        int base = 0;
        for (int j = lane; j < n_keys; j += 32)
            if (s_size[j] > s_size[key] || (s_size[j] == s_size[key] && j < key)) base += s_n[j];
        base = __reduce_add_sync(0xffffffffu, base);
        for (int i = lane; i < s_n[key]; i += 32) {
            FwdWork w;
            w.slice = key;
            w.begin = min(s_seg[key + 1], s_seg[key] + i * s_size[key]);
            w.end = min(s_seg[key + 1], w.begin + s_size[key]);
            w.pad = 0;
            work[base + i] = w;
        }
    }
    if (threadIdx.x < 32) {
        int total = 0;
        for (int j = lane; j < n_keys; j += 32) total += s_n[j];
        total = __reduce_add_sync(0xffffffffu, total);
        if (lane == 0) {
            n_work[0] = total;
            n_work[1] = 0;  // "some item has a row outside its slice", raised by k_fwd_codes
            n_work[2] = 0;  // units taken by the forward's blocks
        }
    }
}

// Chunks of <= ch consecutive slots of one slice, in slice order; groups of <= BWD_GROUP chunks of one slice (an empty slice
// has one group, its rows are zeroed); and per part (equal ranges of slices) the order in which the weight gradient's blocks
// take the groups: the largest first.
static __device__ void plan_backward(const int* __restrict__ s_seg, int n_keys, int ch, int parts, FwdWork* __restrict__ chunks,
                                     int* __restrict__ n_chunks, int* __restrict__ groups, int* __restrict__ sched) {
    __shared__ int s_nc[SORT_MAX_KEYS], s_size[SORT_MAX_KEYS], s_part[SORT_MAX_KEYS];
    __shared__ int s_w[2 * SORT_MAX_KEYS], s_cnt[2 * SORT_MAX_KEYS];  // per slice: its full groups, its last smaller one
    const int n_slices = n_keys - 1;  // the last key holds items without a slice: they have no rows
    const int k = threadIdx.x;
    if (k < n_keys) {
        const int len = s_seg[k + 1] - s_seg[k];
        const int n = (len + ch - 1) / ch;
        s_nc[k] = n;
        const int size = n > 0 ? ((len + n - 1) / n + 7) & ~7 : 0;  // equal chunks (<= ch: ch is a multiple of 8)
        s_size[k] = size;
        if (k < n_slices) {
            const int full = n / BWD_GROUP, rest = n - full * BWD_GROUP;
            s_w[2 * k] = BWD_GROUP * size;
            s_cnt[2 * k] = full;
            s_w[2 * k + 1] = rest * size;
            s_cnt[2 * k + 1] = (rest > 0 || n == 0) ? 1 : 0;
            int p = 0;
            while (p + 1 < parts && k >= (int)((long long)n_slices * (p + 1) / parts)) ++p;
            s_part[k] = p;
        }
    }
    __syncthreads();
    const unsigned all = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    int4* rec = reinterpret_cast<int4*>(groups + 4 + SORT_KEYS_LIMIT + 4);
    int* order = sched + 2 * BWD_PARTS + 4;
    for (int key = threadIdx.x >> 5; key < n_keys; key += PLAN_THREADS / 32) {
        int c0 = 0, g0 = 0, slab = 0;
        int base[2] = {0, 0};  // position of the slice's full groups and of its last smaller one among all groups
        for (int j = lane; j < n_keys; j += 32) {
            if (j < key) c0 += s_nc[j];
            if (j >= n_slices) continue;
            const int ng = s_cnt[2 * j] + s_cnt[2 * j + 1];
            if (j < key) { g0 += ng; slab += ng - 1; }
            if (key < n_slices) {
                for (int h = 0; h < 4; ++h) {
                    const int c = 2 * key + (h & 1), d = 2 * j + (h >> 1);
                    const bool before = s_part[j] != s_part[key] ? s_part[j] < s_part[key] : (s_w[d] > s_w[c] || (s_w[d] == s_w[c] && d < c));
                    if (before) base[h & 1] += s_cnt[d];
                }
            }
        }
        c0 = __reduce_add_sync(all, c0);
        g0 = __reduce_add_sync(all, g0);
        slab = __reduce_add_sync(all, slab);
        base[0] = __reduce_add_sync(all, base[0]);
        base[1] = __reduce_add_sync(all, base[1]);
        const int nc = s_nc[key], size = s_size[key];
        for (int i = lane; i < nc; i += 32) {
            FwdWork w;
            w.slice = key;
            w.begin = min(s_seg[key + 1], s_seg[key] + i * size);
            w.end = min(s_seg[key + 1], w.begin + size);
            w.pad = 0;
            chunks[c0 + i] = w;
        }
        if (lane == 0) {
            groups[4 + key] = g0;  // first group of the slice; of the last key: the end
            if (key == n_slices) {
                *n_chunks = c0 + nc;
                groups[0] = g0;
            }
        }
        if (key < n_slices) {
            const int full = s_cnt[2 * key], ng = full + s_cnt[2 * key + 1];
            for (int i = lane; i < ng; i += 32) {
                rec[g0 + i] = make_int4(key, c0 + min(i * BWD_GROUP, nc), c0 + min((i + 1) * BWD_GROUP, nc), i == 0 ? -1 : slab + i - 1);
                order[i < full ? base[0] + i : base[1] + i - full] = g0 + i;
            }
        }
    }
    if ((int)threadIdx.x <= parts) {  // first position of every part, and the end
        int first = 0;
        for (int j = 0; j < n_slices; ++j)
            if (s_part[j] < (int)threadIdx.x) first += s_cnt[2 * j] + s_cnt[2 * j + 1];
        sched[BWD_PARTS + threadIdx.x] = first;
    }
}

__global__ void __launch_bounds__(PLAN_THREADS) k_step_plans(const int* __restrict__ seg_start, int K0, int ut, TileDesc* __restrict__ tiles,
                                                             int* __restrict__ n_tiles, TileDesc* __restrict__ units, TileDesc* __restrict__ wunits,
                                                             const int* __restrict__ item_seg, int n_keys, FwdWork* __restrict__ work,
                                                             int* __restrict__ n_work, int ch, int parts, FwdWork* __restrict__ chunks,
                                                             int* __restrict__ n_chunks, int* __restrict__ groups, int* __restrict__ sched) {
    __shared__ int s_seg[SORT_MAX_KEYS + 2];
    const int* seg = blockIdx.x == 0 ? seg_start : item_seg;
    const int n = blockIdx.x == 0 ? K0 : n_keys;
    for (int k = threadIdx.x; k <= n; k += PLAN_THREADS) s_seg[k] = seg[k];
    __syncthreads();
    if (blockIdx.x == 0) plan_tiles(s_seg, K0, ut, tiles, n_tiles, units, wunits);
    else if (blockIdx.x == 1) plan_forward(s_seg, n_keys, work, n_work);
    else plan_backward(s_seg, n_keys, ch, parts, chunks, n_chunks, groups, sched);
}

// Positions by bucket and their tiles in one launch of one block, for batches of at most SORT_ONE_BLOCK positions whose items
// need no order: every warp owns a run of positions, counts its keys, and places them behind those of the warps before it.
// (The four launches cost 21 to 24 us however small the batch.)
__global__ void __launch_bounds__(1024) k_sort_one_block(BucketKey fn, int n, int K, int ut, int* __restrict__ order, int* __restrict__ seg_start,
                                                         TileDesc* __restrict__ tiles, int* __restrict__ n_tiles, TileDesc* __restrict__ units,
                                                         TileDesc* __restrict__ wunits) {
    __shared__ int s_cnt[TB_MAX_BUCKETS + 1][32], s_seg[TB_MAX_BUCKETS + 3];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (w < K) s_cnt[w][lane] = 0;
    __syncthreads();
    const int per = ((n + 31) / 32 + 31) & ~31, i0 = w * per, i1 = min(n, i0 + per);
    // place = false: count; the counts are then turned into the first slots
    auto walk = [&](bool place) {
        for (int i = i0; i < i1; i += 32) {
            const bool in = i + lane < i1;
            const int k = in ? fn(i + lane) : K;
            const unsigned same = __match_any_sync(0xffffffffu, k);
            const int before = __popc(same & ((1u << lane) - 1));
            int at = 0;
            if (in) at = s_cnt[k][w] + before;
            __syncwarp();
            if (in && before == 0) s_cnt[k][w] += __popc(same);
            if (in && place) order[at] = i + lane;
            __syncwarp();
        }
    };
    walk(false);
    __syncthreads();
    if (w < K) {
        const int c = s_cnt[w][lane];
        int incl = c;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d) incl += t;
        }
        s_cnt[w][lane] = incl - c;
        if (lane == 31) s_seg[w + 1] = incl;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        s_seg[0] = 0;
        for (int k = 0; k < K; ++k) s_seg[k + 1] += s_seg[k];
    }
    __syncthreads();
    if (w < K) s_cnt[w][lane] += s_seg[w];
    if ((int)threadIdx.x <= K) seg_start[threadIdx.x] = s_seg[threadIdx.x];
    __syncthreads();
    walk(true);
    plan_tiles(s_seg, K, ut, tiles, n_tiles, units, wunits);
}

// The question k_fwd_codes answers for the device, asked as soon as the batch is there, for the host: the slice of an item
// is that of its first feature (ItemKey), slots beyond nnz and indices outside the table do not count.  A warp per position.
__global__ void __launch_bounds__(256) k_slice_check(const int* __restrict__ idx_stm, const int* __restrict__ idx_nstm,
                                                     const int* __restrict__ nnz, int B, int A, int N, int rps, int* outside) {
    const int lane = threadIdx.x & 31;
    bool out = false;
    for (int b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; b < B; b += (gridDim.x * blockDim.x) >> 5) {
        const int n = min(max(nnz[b], 0), A);
        for (int p = 0; p < 2; ++p) {
            const int* ip = (p ? idx_nstm : idx_stm) + (size_t)b * A;
            int slice = 0;
            for (int q = lane; q < ((n + 31) & ~31); q += 32) {
                const int f = q < n ? ip[q] : -1;
                const int k = (unsigned)f < (unsigned)N ? f / rps : -1;
                if (q < 32) slice = __shfl_sync(0xffffffffu, k, 0);
                out = out || (k >= 0 && k != slice);
            }
        }
    }
    if (out) *outside = 1;
}

int launch_slice_check(cudaStream_t s, const int* idx_stm, const int* idx_nstm, const int* nnz, int B, int A, int N, int rows_per_slice,
                       int* outside) {
    if (B <= 0) return 0;
    const int blocks = ceil_div(B, 8);
    k_slice_check<<<blocks < 8 * sm_count() ? blocks : 8 * sm_count(), 256, 0, s>>>(idx_stm, idx_nstm, nnz, B, A, N, rows_per_slice, outside);
    return 1;
}

int sort_weight_units(int n_pos) { return n_pos / (TB_UNIT_TILES * TB_TILE_M) + TB_MAX_BUCKETS + 2; }
int sort_units(int n_pos) { return n_pos / (unit_tiles(n_pos) * TB_TILE_M) + TB_MAX_BUCKETS + 2; }
// at least a unit per SM: batches with smaller units have no more (unit_tiles)
int sort_max_units(int max_tiles) {
    const int sms = sm_count(), n = max_tiles / TB_UNIT_TILES > sms ? max_tiles / TB_UNIT_TILES : sms;
    return n + TB_MAX_BUCKETS + 2;
}

const TileDesc* weight_units(const TileDesc* tiles, int max_tiles) { return tiles + max_tiles + sort_max_units(max_tiles); }
size_t sort_tiles_len(int max_tiles) { return (size_t)max_tiles + sort_max_units(max_tiles) + max_tiles / TB_UNIT_TILES + TB_MAX_BUCKETS + 2; }

// Both sorts of a step in four launches: positions by bucket (order, tiles, units) and items by table slice, with the plans
// of the slice-resident kernels where their work buffers are given; without `items` (B <= SORT_ONE_BLOCK) the positions alone,
// in one launch.
// hist: scratch of (nb + 1) * ceil(B / 1024) + (slices + 1) * ceil(n_persp * B / 1024) ints.
int launch_step_sorts(cudaStream_t s, const int* bucket, int B, int nb, int* order, TileDesc* tiles, int* n_tiles, int* seg_start,
                      int max_tiles, const int* idx_stm, const int* idx_nstm, const int* nnz, int A, int N, int rows_per_slice,
                      int n_persp, int* items, int* item_seg, int* hist, int* fwd_work, int* bwd_work, int bwd_parts) {
    int n_slices = ceil_div(N, rows_per_slice);
    if (n_slices + 1 > SORT_MAX_KEYS) {
        rows_per_slice = ceil_div(N, SORT_MAX_KEYS - 1);
        n_slices = ceil_div(N, rows_per_slice);
    }
    const int K0 = nb + 1, G0 = ceil_div(B, SORT_BLOCK);
    if (!items) {
        k_sort_one_block<<<1, 1024, 0, s>>>(BucketKey{bucket, nb}, B, K0, unit_tiles(B), order, seg_start, tiles, n_tiles, tiles + max_tiles,
                                             const_cast<TileDesc*>(weight_units(tiles, max_tiles)));
        return 1;
    }
    const int n1 = n_persp * B, K1 = n_slices + 1, G1 = ceil_div(n1, SORT_BLOCK);
    int* h0 = hist;
    int* h1 = hist + (size_t)K0 * G0;
    BucketKey f0{bucket, nb};
    ItemKey f1{idx_stm, idx_nstm, nnz, B, A, N, rows_per_slice, n_slices};
    const dim3 grid(G0 > G1 ? G0 : G1, 2);
    k_sort_hist2<<<grid, SORT_BLOCK, 0, s>>>(f0, B, K0, G0, h0, f1, n1, K1, G1, h1);
    k_sort_scan2<<<2, 1024, 0, s>>>(h0, K0, G0, B, seg_start, h1, K1, G1, n1, item_seg);
    k_sort_scatter2<<<grid, SORT_BLOCK, 0, s>>>(f0, B, K0, G0, h0, order, f1, n1, K1, G1, h1, items);
    SliceBuffers sb = {};
    BwdPointers bp = {};
    int ch = 0;
    if (fwd_work) sb = slice_buffers(fwd_work, n1, K1);
    if (bwd_work) {
        const BwdLayout L = bwd_layout(n1, A, rows_per_slice);
        bp = bwd_pointers(bwd_work, L);
        ch = L.CH;
    }
    k_step_plans<<<bwd_work ? 3 : fwd_work ? 2 : 1, PLAN_THREADS, 0, s>>>(seg_start, K0, unit_tiles(B), tiles, n_tiles, tiles + max_tiles,
                                                                          const_cast<TileDesc*>(weight_units(tiles, max_tiles)), item_seg, K1,
                                                                          sb.work, sb.n_work, ch, bwd_parts, bp.chunks, bp.n_chunks,
                                                                          bp.groups, bp.sched);
    return 4;
}
