// Sparse feature-transformer kernels: forward gather-sum (fused with the FT activation), inverse
// index, backward segmented reduce, factorizer reduce / fold.
//
// Layout: the FT table is row-major [rows, F] f32 (w[f*F + c], native_kernels.cu:162-200); every
// per-position tensor is row-major [B, F].  F is a multiple of 128, so rows are 512-byte aligned and
// every access below is a 128-bit vector.
#include "common.cuh"
#include "ft_slice.cuh"
#include <stdlib.h>

#define SORT_KEYS_MAX 128  // key limit of the small-key sorts (sort_kernels.cu)

// ------------------------------------------------------------------------------------------------
// forward: one (position, perspective) item per group of F/8 threads.  Thread `lane` owns the float4
// at column 4*lane and its pair partner at column F/2 + 4*lane, so that the pairwise product of the
// LayerStack activation never leaves the thread.  Rows are added in slot order with plain f32 adds:
// the sums are bit-identical to sparse_ft_forward_cpu (sparse/sparse_ft_forward.rs:54-78).
// ------------------------------------------------------------------------------------------------
// four consecutive table / activation values as fp32, whatever their storage type
template <bool H>
static __device__ __forceinline__ float4 ld4(const void* base, size_t elem) {
    if (H) {
        const uint2 u = __ldg(reinterpret_cast<const uint2*>(static_cast<const __half*>(base) + elem));
        const float2 a = unpack_h2(u.x), b = unpack_h2(u.y);
        return make_float4(a.x, a.y, b.x, b.y);
    }
    return __ldg(reinterpret_cast<const float4*>(static_cast<const float*>(base) + elem));
}
template <bool H>
static __device__ __forceinline__ void st4_cs(void* base, size_t elem, float4 v) {
    if (H) __stcs(reinterpret_cast<uint2*>(static_cast<__half*>(base) + elem), make_uint2(pack_h2(v.x, v.y), pack_h2(v.z, v.w)));
    else __stcs(reinterpret_cast<float4*>(static_cast<float*>(base) + elem), v);
}
static __device__ __forceinline__ float4 round_h4(float4 v) {
    const float2 a = unpack_h2(pack_h2(v.x, v.y)), b = unpack_h2(pack_h2(v.z, v.w));
    return make_float4(a.x, a.y, b.x, b.y);
}

// TH: fp16 table rows (summed in fp32); OH: fp16 pre-activations, the activation computed from the rounded values
template <int MODE, bool TH, bool OH>
__global__ void __launch_bounds__(512) k_ft_forward(const void* __restrict__ table, const int* __restrict__ idx_stm,
                                                     const int* __restrict__ idx_nstm, const int* __restrict__ nnz,
                                                     const float* __restrict__ bias, void* __restrict__ pre_stm,
                                                     void* __restrict__ pre_nstm, float* __restrict__ combined,
                                                     const int* __restrict__ items, int n_items, int B, int F, int N, int A,
                                                     float scale, int ipc) {
    extern __shared__ int s_idx[];  // [ipc][A] indices, then [ipc] item ids
    int* s_item = s_idx + ipc * A;
    const int tpi = F >> 3;
    const int il = threadIdx.x / tpi;
    const int lane = threadIdx.x - il * tpi;
    const int slot0 = blockIdx.x * ipc;

    for (int i = threadIdx.x; i < ipc; i += blockDim.x) {
        const int sl = slot0 + i;
        s_item[i] = sl < n_items ? (items ? items[sl] : sl) : -1;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < ipc * A; i += blockDim.x) {
        const int li = i / A, a = i - li * A;
        const int it = s_item[li];
        int v = -1;
        if (it >= 0) {
            const int p = it >= B, b = it - p * B;
            if (a < nnz[b]) v = (p ? idx_nstm : idx_stm)[(size_t)b * A + a];
        }
        if ((unsigned)v >= (unsigned)N) v = -1;  // padding and out-of-range indices are skipped
        s_idx[i] = v;
    }
    __syncthreads();
    const int it = s_item[il];
    if (it < 0) return;
    const int persp = it >= B;
    const int item = it - persp * B;  // the position
    int n = nnz[item];
    n = n < 0 ? 0 : (n > A ? A : n);
    const int* my = s_idx + il * A;
    const int row4 = F >> 2;
    const int c0 = lane, c1 = lane + tpi;

    float4 acc0 = make_float4(0.f, 0.f, 0.f, 0.f), acc1 = acc0;
    for (int a0 = 0; a0 < n; a0 += 8) {
        float4 va[8], vb[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int f = (a0 + u < n) ? my[a0 + u] : -1;
            if (f >= 0) {
                va[u] = ld4<TH>(table, (size_t)f * F + 4 * c0);
                vb[u] = ld4<TH>(table, (size_t)f * F + 4 * c1);
            } else {
                va[u] = make_float4(0.f, 0.f, 0.f, 0.f);  // x + 0.0 == x: a skipped slot leaves the sum unchanged
                vb[u] = va[u];
            }
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            acc0.x += va[u].x; acc0.y += va[u].y; acc0.z += va[u].z; acc0.w += va[u].w;
            acc1.x += vb[u].x; acc1.y += vb[u].y; acc1.z += vb[u].z; acc1.w += vb[u].w;
        }
    }

    void* pre = persp ? pre_nstm : pre_stm;
    const size_t e0 = (size_t)item * F + 4 * c0, e1 = (size_t)item * F + 4 * c1;
    if (OH) { acc0 = round_h4(acc0); acc1 = round_h4(acc1); }
    // outputs are written once and read by later kernels only: streaming stores leave L2 to the table slice
    if (MODE == 0) {
        st4_cs<OH>(pre, e0, acc0);
        st4_cs<OH>(pre, e1, acc1);
    } else if (MODE == 1) {
        // ft_post_perspective_fwd (layerstack/ft_post_perspective.rs:57-83): the raw sums are kept for the
        // backward pass, combined[b, persp*F/2 + r] = crelu(x_r + b_r) * crelu(x_{r+F/2} + b_{r+F/2}) * scale
        st4_cs<OH>(pre, e0, acc0);
        st4_cs<OH>(pre, e1, acc1);
        const float4 b0 = __ldg(reinterpret_cast<const float4*>(bias) + c0);
        const float4 b1 = __ldg(reinterpret_cast<const float4*>(bias) + c1);
        float4 o;
        o.x = crelu01(acc0.x + b0.x) * crelu01(acc1.x + b1.x) * scale;
        o.y = crelu01(acc0.y + b0.y) * crelu01(acc1.y + b1.y) * scale;
        o.z = crelu01(acc0.z + b0.z) * crelu01(acc1.z + b1.z) * scale;
        o.w = crelu01(acc0.w + b0.w) * crelu01(acc1.w + b1.w) * scale;
        __stcs(reinterpret_cast<float4*>(combined) + (size_t)item * row4 + persp * tpi + c0, o);
    } else {
        // simple_ft_post_fused_{crelu,screlu} (native_kernels.cu:1406-1450): the biased value replaces the
        // raw sum, combined[b, persp*F + c] = act(x)
        const float4 b0 = __ldg(reinterpret_cast<const float4*>(bias) + c0);
        const float4 b1 = __ldg(reinterpret_cast<const float4*>(bias) + c1);
        float4 x0 = make_float4(acc0.x + b0.x, acc0.y + b0.y, acc0.z + b0.z, acc0.w + b0.w);
        float4 x1 = make_float4(acc1.x + b1.x, acc1.y + b1.y, acc1.z + b1.z, acc1.w + b1.w);
        st4_cs<OH>(pre, e0, x0);
        st4_cs<OH>(pre, e1, x1);
        float4 a0 = make_float4(crelu01(x0.x), crelu01(x0.y), crelu01(x0.z), crelu01(x0.w));
        float4 a1 = make_float4(crelu01(x1.x), crelu01(x1.y), crelu01(x1.z), crelu01(x1.w));
        if (MODE == 3) {
            a0.x *= a0.x; a0.y *= a0.y; a0.z *= a0.z; a0.w *= a0.w;
            a1.x *= a1.x; a1.y *= a1.y; a1.z *= a1.z; a1.w *= a1.w;
        }
        float4* comb = reinterpret_cast<float4*>(combined) + (size_t)item * (2 * row4) + persp * row4;
        __stcs(comb + c0, a0);
        __stcs(comb + c1, a1);
    }
}

int launch_ft_forward(cudaStream_t s, int mode, const void* table, const int* idx_stm, const int* idx_nstm,
                      const int* nnz, const float* bias, void* pre_stm, void* pre_nstm, float* combined,
                      const int* items, int B, int F, int N, int A, float scale, int n_persp, int table_half, int out_half) {
    if (B <= 0) return 0;
    const int tpi = F / 8;
    int ipc = 256 / tpi;
    if (ipc < 1) ipc = 1;
    const int n_items = n_persp * B;
    dim3 grid(ceil_div(n_items, ipc)), block(ipc * tpi);
    size_t smem = (size_t)ipc * (A + 1) * sizeof(int);
#define FT_FWD_ARGS table, idx_stm, idx_nstm, nnz, bias, pre_stm, pre_nstm, combined, items, n_items, B, F, N, A, scale, ipc
    if (table_half) {
        if (mode == 1 && !out_half) k_ft_forward<1, true, false><<<grid, block, smem, s>>>(FT_FWD_ARGS);
        else if (mode == 1) k_ft_forward<1, true, true><<<grid, block, smem, s>>>(FT_FWD_ARGS);
        else return -1;
        return 1;
    }
    if (out_half) return -1;
    switch (mode) {
        case 0: k_ft_forward<0, false, false><<<grid, block, smem, s>>>(FT_FWD_ARGS); break;
        case 1: k_ft_forward<1, false, false><<<grid, block, smem, s>>>(FT_FWD_ARGS); break;
        case 2: k_ft_forward<2, false, false><<<grid, block, smem, s>>>(FT_FWD_ARGS); break;
        default: k_ft_forward<3, false, false><<<grid, block, smem, s>>>(FT_FWD_ARGS); break;
    }
#undef FT_FWD_ARGS
    return 1;
}

// ------------------------------------------------------------------------------------------------
// forward, slice-resident variant.  The generic kernel above gathers every row from L2; with the items sorted
// by king-bucket slice all of an item's rows lie in one slice of rows_per_slice rows, and a 32-column strip
// of that slice (rows_per_slice * 128 bytes, 208 KB for 1629 rows) fits in shared memory.  A block owns
// (run of <= SLICE_IPC items of one slice, column strip), loads the strip once and serves all of its items'
// row reads from shared memory; eight lanes work on one item, a lane on four adjacent columns (128-bit
// shared loads), rows are added in slot order as in the generic kernel, so the sums are bit-identical.
// A row outside the block's slice (arbitrary index lists) is read from the table in global memory instead.
// LayerStack strips hold columns [16s, 16s+16) and their pair partners [F/2 + 16s, F/2 + 16s + 16); the other
// modes 32 adjacent columns.
// ------------------------------------------------------------------------------------------------
// Row codes of the slice-resident forward, for every slot of the sorted item list: per feature slot the
// row number inside the item's slice (16 bits), rps for a slot without a feature (the strip
// keeps a row of zeros there), SLICE_OUTSIDE for a table row outside the slice (the kernel then reads the index list).
// info[slot] = item | SLICE_SLOW_BIT when the item has an outside row.  Codes of consecutive slots are contiguous
// (A_pad 16-bit codes each, A_pad a multiple of 8), so a warp copies its round of four items in 16-byte pieces.
// A thread does eight cells (the lanes of a slot sit in one warp): the kernel is a chain of dependent loads, so what counts
// is how many of them run side by side (a thread per slot: 8.4 us at 2048 items, 20 at 131 072).
__global__ void __launch_bounds__(256) k_fwd_codes(const int* __restrict__ idx_stm, const int* __restrict__ idx_nstm,
                                                   const int* __restrict__ nnz, const int* __restrict__ items,
                                                   const int* __restrict__ item_seg, int n_keys, int n_items, int B, int N,
                                                   int A, int A_pad, int rps, uint4* __restrict__ codes,
                                                   int* __restrict__ info, int* __restrict__ outside_flag) {
    __shared__ int s_seg[SORT_KEYS_MAX + 2];
    for (int k = threadIdx.x; k <= n_keys; k += blockDim.x) s_seg[k] = item_seg[k];
    __syncthreads();
    const int per = A_pad >> 3, slots_per_warp = 32 / per;
    const int lane = threadIdx.x & 31, warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int li = lane / per, part = lane - li * per;
    const int s = warp * slots_per_warp + li;
    const bool live = li < slots_per_warp && s < n_items;
    bool outside = false;
    int it = 0;
    if (live) {
        it = __ldg(items + s);
        int lo = 0, hi = n_keys - 1;  // the key whose segment holds slot s
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (s_seg[mid] <= s) lo = mid; else hi = mid - 1;
        }
        const int row0 = lo * rps;
        const int rows = max(0, min(rps, N - row0));
        const int p = it >= B, b = it - p * B;
        int n = __ldg(nnz + b);
        n = n < 0 ? 0 : (n > A ? A : n);
        const int* ip = (p ? idx_nstm : idx_stm) + (size_t)b * A;
        const int q0 = 8 * part;
        unsigned c[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int q = q0 + u;
            unsigned code = (unsigned)rps;
            if (q < n) {
                const int f = __ldg(ip + q);
                if ((unsigned)f < (unsigned)N) {
                    const int r = f - row0;
                    if ((unsigned)r < (unsigned)rows) code = (unsigned)r;
                    else { code = SLICE_OUTSIDE; outside = true; }
                }
            }
            c[u] = code;
        }
        codes[((size_t)s * A_pad + q0) >> 3] = make_uint4(c[0] | (c[1] << 16), c[2] | (c[3] << 16), c[4] | (c[5] << 16), c[6] | (c[7] << 16));
    }
    const unsigned out = __ballot_sync(0xffffffffu, outside) >> (li * per) & ((1u << per) - 1u);
    if (live && part == 0) {
        info[s] = it | (out ? SLICE_SLOW_BIT : 0);
        if (out) *outside_flag = 1;
    }
}

// TH: the table holds fp16 rows (the strip is then 64 columns wide: a lane reads 16 bytes = eight columns of every row and
// sums them in fp32, native_kernels.cu:743-801 sparse_ft_forward_fp16); OH: the pre-activations are stored as fp16 and the
// activation is computed from the rounded value (sparse_ft_forward_fp16_out + ft_post_perspective_fwd_fp16, :837-863).
// Persistent: one block per SM takes (run, strip) units from a counter, the runs largest first (k_step_plans).  (Prefetching
// the next unit's strip into L2 meanwhile cost 1.5 %.)
template <int MODE, bool TH, bool OH>
__global__ void __launch_bounds__(1024, 1) k_ft_forward_slice(const void* __restrict__ table_v, const float* __restrict__ bias,
                                                               void* __restrict__ pre_stm_v, void* __restrict__ pre_nstm_v,
                                                               float* __restrict__ combined, const int* __restrict__ idx_stm,
                                                               const int* __restrict__ idx_nstm, const int* __restrict__ info,
                                                               const uint4* __restrict__ codes, const FwdWork* __restrict__ work,
                                                               int* __restrict__ n_work, int strips, int B, int F, int N,
                                                               int A, int A_pad, int rps, float scale) {
    constexpr int W = TH ? 8 : 4;          // columns per lane
    constexpr int TSZ = TH ? 2 : 4;        // bytes per table element
    constexpr int OSZ = OH ? 2 : 4;        // bytes per stored pre-activation
    // strip [rps + 1][8 W] elements (128 bytes per row), then two buffers of [warps][4 items][A_pad] 16-bit row codes
    extern __shared__ __align__(16) unsigned char s_raw[];
    __shared__ int s_unit;
    const int half = F >> 1;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 3, j = lane & 7;
    const unsigned char* __restrict__ table = static_cast<const unsigned char*>(table_v);
    const int n_units = n_work[0] * strips;
    // a round = four items per warp; their codes arrive by asynchronous copy one round ahead
    const int code_bytes = 4 * A_pad * 2;  // per warp and buffer
    const int buf_stride = (blockDim.x >> 5) * code_bytes;
    unsigned char* s_codes = s_raw + ((size_t)rps + 1) * 128 + (size_t)warp * code_bytes;
    const unsigned char* codes_b = reinterpret_cast<const unsigned char*>(codes);
    const int chunk_item = (lane * 16) / (A_pad * 2);  // which of the four items this lane's 16-byte piece belongs to
    const int per_round = 4 * (blockDim.x >> 5);
    const unsigned char* s_lane = s_raw + 16 * j;
    if (threadIdx.x < 32) reinterpret_cast<float*>(s_raw)[rps * 32 + threadIdx.x] = 0.f;  // the row of zeros
    auto first_col = [&](int strip, int jj) {  // of the lanes with column index jj
        return MODE == 1 ? (jj < 4 ? 4 * W * strip + W * jj : half + 4 * W * strip + W * (jj - 4)) : 8 * W * strip + W * jj;
    };

    // the first units go by block number (the counter starts behind them)
    for (int unit = blockIdx.x; unit < n_units;) {
    const FwdWork wk = work[unit / strips];
    const int strip = unit % strips;
    const int row0 = wk.slice * rps;
    const int rows = max(0, min(rps, N - row0));
    const int mycol = first_col(strip, j);

    // strip fill: thread e & 7 == j copies the 16 bytes it will later read, for rows e >> 3
    for (int e = threadIdx.x; e < rows * 8; e += blockDim.x)
        cp_async16(s_raw + (size_t)e * 16, table + ((size_t)(row0 + (e >> 3)) * F + mycol) * TSZ, 16);
    cp_async_commit();
    if (threadIdx.x == 0) s_unit = (int)gridDim.x + atomicAdd(n_work + 2, 1);
    for (int e = rows * 8 + threadIdx.x; e < rps * 8; e += blockDim.x)  // rows past the end of the table
        *reinterpret_cast<float4*>(s_raw + (size_t)e * 16) = make_float4(0.f, 0.f, 0.f, 0.f);
    auto fetch_codes = [&](int slot, int bf) {
        if (lane * 16 < code_bytes) {
            const bool ok = slot + chunk_item < wk.end;
            const long long off = (long long)slot * A_pad * 2 + lane * 16;
            cp_async16(s_codes + bf * buf_stride + lane * 16, codes_b + (ok ? off : 0), ok ? 16 : 0);
        }
    };
    int buf = 0;
    fetch_codes(wk.begin + 4 * warp, 0);
    cp_async_commit();
    auto fetch_info = [&](int slot) { return slot < wk.end ? __ldg(info + slot) : -1; };
    int info_reg = fetch_info(wk.begin + 4 * warp + g);
    cp_async_wait<0>();
    __syncthreads();
    const int next_unit = s_unit;

    // fp32 lanes keep the bias of their four columns and of the pair partner's in registers; fp16 lanes (eight columns)
    // read it in the epilogue instead (L1 hits), their registers are taken by the wider running sums
    float4 mybias = make_float4(0.f, 0.f, 0.f, 0.f);
    if (!TH && bias) mybias = *reinterpret_cast<const float4*>(bias + mycol);
    float4 pbias = mybias;  // the pair partner's bias (LayerStack)
    pbias.x = __shfl_xor_sync(0xffffffffu, mybias.x, 4); pbias.y = __shfl_xor_sync(0xffffffffu, mybias.y, 4);
    pbias.z = __shfl_xor_sync(0xffffffffu, mybias.z, 4); pbias.w = __shfl_xor_sync(0xffffffffu, mybias.w, 4);

    for (int base = wk.begin; base < wk.end; base += per_round) {
        const int inf = info_reg;
        fetch_codes(base + per_round + 4 * warp, buf ^ 1);
        cp_async_commit();
        cp_async_wait<1>();
        __syncwarp();
        info_reg = fetch_info(base + per_round + 4 * warp + g);
        const bool slow = __any_sync(0xffffffffu, inf >= 0 && (inf & SLICE_SLOW_BIT));
        const int it_c = inf < 0 ? -1 : (inf & ~SLICE_SLOW_BIT);
        const unsigned char* my_codes = s_codes + buf * buf_stride + g * A_pad * 2;
        buf ^= 1;

        LaneAcc<TH> acc;
        acc.zero();
        if (!slow) {
            // every row of the round comes from the strip: branch-free; a slot without a feature reads the row of zeros
            // (x + 0.0 == x), rows are added in slot order
#pragma unroll 1
            for (int q = 0; q < A_pad; q += 8) {
                const uint4 c = *reinterpret_cast<const uint4*>(my_codes + 2 * q);
                const ulonglong2 v0 = *reinterpret_cast<const ulonglong2*>(s_lane + (c.x & 0xffffu) * 128u);
                const ulonglong2 v1 = *reinterpret_cast<const ulonglong2*>(s_lane + (c.x >> 16) * 128u);
                const ulonglong2 v2 = *reinterpret_cast<const ulonglong2*>(s_lane + (c.y & 0xffffu) * 128u);
                const ulonglong2 v3 = *reinterpret_cast<const ulonglong2*>(s_lane + (c.y >> 16) * 128u);
                const ulonglong2 v4 = *reinterpret_cast<const ulonglong2*>(s_lane + (c.z & 0xffffu) * 128u);
                const ulonglong2 v5 = *reinterpret_cast<const ulonglong2*>(s_lane + (c.z >> 16) * 128u);
                const ulonglong2 v6 = *reinterpret_cast<const ulonglong2*>(s_lane + (c.w & 0xffffu) * 128u);
                const ulonglong2 v7 = *reinterpret_cast<const ulonglong2*>(s_lane + (c.w >> 16) * 128u);
                acc.add(v0); acc.add(v1); acc.add(v2); acc.add(v3);
                acc.add(v4); acc.add(v5); acc.add(v6); acc.add(v7);
            }
        } else {
            const int p = it_c >= B, bb = it_c < 0 ? 0 : it_c - p * B;
            const int* ip = (p ? idx_nstm : idx_stm) + (size_t)bb * A;
            for (int q = 0; q < A_pad; ++q) {
                const unsigned c = reinterpret_cast<const unsigned short*>(my_codes)[q];
                ulonglong2 v;
                if (c != SLICE_OUTSIDE || it_c < 0) v = *reinterpret_cast<const ulonglong2*>(s_lane + min(c, (unsigned)rps) * 128u);
                else v = __ldg(reinterpret_cast<const ulonglong2*>(table + ((size_t)__ldg(ip + q) * F + mycol) * TSZ));
                acc.add(v);
            }
        }
        __syncwarp();  // all lanes are done with this round's codes before the next round's replace them

        // ---- epilogue: x[] = the lane's sums as the later kernels will read them (rounded to fp16 when stored so)
        float x[W];
#pragma unroll
        for (int i = 0; i < W; ++i) x[i] = acc.get(i);
        const bool valid = it_c >= 0;
        const int persp = it_c >= B, b = valid ? it_c - persp * B : 0;
        unsigned char* pre = static_cast<unsigned char*>(persp ? pre_nstm_v : pre_stm_v) + ((size_t)b * F + mycol) * OSZ;
        auto store_pre = [&](const float* val) {
            if (OH) {
                unsigned h[W / 2];
#pragma unroll
                for (int i = 0; i < W / 2; ++i) h[i] = pack_h2(val[2 * i], val[2 * i + 1]);
                if (W == 8) __stcs(reinterpret_cast<uint4*>(pre), make_uint4(h[0], h[1], h[W / 2 - 2], h[W / 2 - 1]));
                else __stcs(reinterpret_cast<uint2*>(pre), make_uint2(h[0], h[1]));
            } else {
#pragma unroll
                for (int i = 0; i < W; i += 4) __stcs(reinterpret_cast<float4*>(pre) + i / 4, make_float4(val[i], val[i + 1], val[i + 2], val[i + 3]));
            }
        };
        if (OH) {
#pragma unroll
            for (int i = 0; i < W; i += 2) {
                const float2 r = unpack_h2(pack_h2(x[i], x[i + 1]));
                x[i] = r.x; x[i + 1] = r.y;
            }
        }
        if (MODE == 0) {
            if (valid) store_pre(x);
        } else if (MODE == 1) {
            float px[W];  // the pair partner's values
#pragma unroll
            for (int i = 0; i < W; ++i) px[i] = __shfl_xor_sync(0xffffffffu, x[i], 4);
            if (valid) {
                store_pre(x);
                if (j < 4) {
                    float o[W], bm[W], bp[W];
                    if (TH) {
#pragma unroll
                        for (int i = 0; i < W; i += 4) {
                            const float4 u = __ldg(reinterpret_cast<const float4*>(bias + mycol + i));
                            const float4 w = __ldg(reinterpret_cast<const float4*>(bias + half + mycol + i));
                            bm[i] = u.x; bm[i + 1] = u.y; bm[i + 2] = u.z; bm[i + 3] = u.w;
                            bp[i] = w.x; bp[i + 1] = w.y; bp[i + 2] = w.z; bp[i + 3] = w.w;
                        }
                    } else {
                        bm[0] = mybias.x; bm[1] = mybias.y; bm[2] = mybias.z; bm[3] = mybias.w;
                        bp[0] = pbias.x; bp[1] = pbias.y; bp[2] = pbias.z; bp[3] = pbias.w;
                    }
#pragma unroll
                    for (int i = 0; i < W; ++i) o[i] = crelu01(x[i] + bm[i]) * crelu01(px[i] + bp[i]) * scale;
                    float4* dst = reinterpret_cast<float4*>(combined + (size_t)b * F + persp * half + mycol);
#pragma unroll
                    for (int i = 0; i < W; i += 4) __stcs(dst + i / 4, make_float4(o[i], o[i + 1], o[i + 2], o[i + 3]));
                }
            }
        } else if (valid) {
            float y[W], a[W];
            const float bz[4] = {mybias.x, mybias.y, mybias.z, mybias.w};
#pragma unroll
            for (int i = 0; i < W; ++i) {
                y[i] = x[i] + (TH ? __ldg(bias + mycol + i) : bz[i & 3]);
                a[i] = crelu01(y[i]);
                if (MODE == 3) a[i] *= a[i];
            }
            store_pre(y);
            float4* dst = reinterpret_cast<float4*>(combined + (size_t)b * 2 * F + persp * F + mycol);
#pragma unroll
            for (int i = 0; i < W; i += 4) __stcs(dst + i / 4, make_float4(a[i], a[i + 1], a[i + 2], a[i + 3]));
        }
    }
    cp_async_wait<0>();
    __syncthreads();  // the strip has been read by all, s_unit too
    unit = next_unit;
    }
}


// work: FwdWork records, one int (their count), the slot info [n_items], then the 16-bit row codes [n_items][A rounded up to 8]
size_t ft_forward_slice_work_ints(int n_items, int n_keys, int A) {
    return 4 * slice_max_work(n_items, n_keys) + 4 + ((size_t)n_items + 3) / 4 * 4 + ((size_t)n_items * slice_a_pad(A) + 1) / 2 + 4;
}

// Warps of a block: 32, or what the shared memory beside the strip has room for (the sets of 1710 rows leave room for the
// codes of 20: the shared-memory pipe, not the number of warps, sets the pace).  0: the strip does not fit.
static inline int slice_warps(int rps, int A) {
    const long long room = 227 * 1024 - 1024 - ((long long)rps + 1) * 128, per_warp = 2 * 4 * slice_a_pad(A) * 2;
    const long long w = room / per_warp;
    return w < 12 ? 0 : w > 32 ? 32 : (int)w;
}
static inline size_t slice_smem_bytes(int rps, int A) { return ((size_t)rps + 1) * 128 + (size_t)slice_warps(rps, A) * 2 * 4 * slice_a_pad(A) * 2; }

bool ft_forward_slice_supported(int F, int N, int A, int rps) {
    int n_slices = ceil_div(N, rps);
    return F % 128 == 0 && A <= 64 && rps < 0xFFFF && slice_warps(rps, A) > 0 && n_slices + 1 <= SORT_KEYS_MAX;
}

int launch_ft_forward_slice(cudaStream_t s, int mode, const void* table, const int* idx_stm, const int* idx_nstm,
                            const int* nnz, const float* bias, void* pre_stm, void* pre_nstm, float* combined,
                            const int* items, const int* item_seg, int* work, int B, int F, int N, int A, int rps,
                            float scale, int n_persp, int table_half, int out_half) {
    if (B <= 0) return 0;
    const int n_items = n_persp * B;
    const int n_slices = ceil_div(N, rps), n_keys = n_slices + 1;
    const int A_pad = slice_a_pad(A);
    const SliceBuffers sb = slice_buffers(work, n_items, n_keys);
    FwdWork* wk = sb.work;
    int* n_work = sb.n_work;
    int* info = sb.info;
    uint4* codes = sb.codes;
    const int slots_per_block = 8 * (32 / (A_pad / 8));
    k_fwd_codes<<<ceil_div(n_items, slots_per_block), 256, 0, s>>>(idx_stm, idx_nstm, nnz, items, item_seg, n_keys, n_items, B, N, A, A_pad,
                                                       rps, codes, info, sb.outside_flag);
    const size_t smem = slice_smem_bytes(rps, A);
    const int strips = table_half ? F / 64 : F / 32, grid = sm_count(), threads = 32 * slice_warps(rps, A);
#define FT_SLICE_LAUNCH(M, TH, OH)                                                                                       \
    do {                                                                                                                 \
        cudaFuncSetAttribute(k_ft_forward_slice<M, TH, OH>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);     \
        k_ft_forward_slice<M, TH, OH><<<grid, threads, smem, s>>>(table, bias, pre_stm, pre_nstm, combined, idx_stm, idx_nstm, \
                                                               info, codes, wk, n_work, strips, B, F, N, A, A_pad, rps, \
                                                               scale);                                                   \
    } while (0)
    if (table_half) {  // fp16 table: the LayerStack activation, with fp32 or fp16 pre-activations
        if (mode == 1 && !out_half) FT_SLICE_LAUNCH(1, true, false);
        else if (mode == 1) FT_SLICE_LAUNCH(1, true, true);
        else return -1;
    } else {
        if (out_half) return -1;
        switch (mode) {
            case 0: FT_SLICE_LAUNCH(0, false, false); break;
            case 1: FT_SLICE_LAUNCH(1, false, false); break;
            case 2: FT_SLICE_LAUNCH(2, false, false); break;
            default: FT_SLICE_LAUNCH(3, false, false); break;
        }
    }
#undef FT_SLICE_LAUNCH
    return 2;
}

// ------------------------------------------------------------------------------------------------
// inverse index: for every feature the list of positions that hold it (the counting sort of
// native_kernels.cu:1630-1765: histogram, offsets, ranked scatter).
//
// The histogram's atomics hand out the ranks, so the scatter needs none.  The lists lie in the order in which the scan's
// blocks take their room (an atomic per block of SCAN_CELLS rows): nothing needs them in row order, and one launch does
// what a scan over all blocks took two for.  Its threads also plan the gradient: long lists are queued for sorting, very
// long ones cut into parts.
// ------------------------------------------------------------------------------------------------
// counters behind the histogram
#define INV_ROOM 0   // [2] list cells taken so far, per perspective
#define INV_QUEUED 2 // lists queued for k_lists_sort_long
#define INV_PARTS 3  // parts of split rows
#define INV_SPLIT 4  // split rows
#define INV_COUNTERS 5

// the unsigned 32-bit indices hold every list cell: batch * slots is an int everywhere else as well
__global__ void __launch_bounds__(256) k_feat_count(const int* __restrict__ idx_stm, const int* __restrict__ idx_nstm,
                                                    const int* __restrict__ nnz, unsigned cells, unsigned A, int N,
                                                    int* __restrict__ counts, int* __restrict__ ranks) {
    const int* idx = blockIdx.y ? idx_nstm : idx_stm;
    int* cnt = counts + (size_t)blockIdx.y * N;
    int* rank = ranks + (size_t)blockIdx.y * cells;
    for (unsigned r = blockIdx.x * 256 + threadIdx.x; r < cells; r += gridDim.x * 256) {
        const unsigned b = r / A, a = r - b * A;
        const int f = idx[r];
        if ((int)a < nnz[b] && (unsigned)f < (unsigned)N) rank[r] = atomicAdd(cnt + f, 1);
    }
}

#define SCAN_CELLS 2048
#define BWD_PART 4096  // entries (both perspectives) from which a row is summed in parts
__global__ void __launch_bounds__(1024) k_feat_scan(const int* __restrict__ counts, int N, int n_persp, int sort_limit,
                                                    int* __restrict__ offsets, int* __restrict__ counters,
                                                    int* __restrict__ long_queue, int2* __restrict__ work, int* __restrict__ split) {
    __shared__ int s_warp[32], s_base;
    const int p = blockIdx.y;
    const int* c = counts + (size_t)p * N;
    int* o = offsets + (size_t)p * N;
    const int i0 = blockIdx.x * SCAN_CELLS + 2 * threadIdx.x;
    const int n0 = i0 < N ? c[i0] : 0, n1 = i0 + 1 < N ? c[i0 + 1] : 0;
    const int sum = n0 + n1;
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
        if (lane == 31) s_base = atomicAdd(counters + INV_ROOM + p, ti);
    }
    __syncthreads();
    const int excl = s_base + s_warp[w] + incl - sum;
    if (i0 < N) o[i0] = excl;
    if (i0 + 1 < N) o[i0 + 1] = excl + n0;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const int f = i0 + k, n = k ? n1 : n0;
        if (f >= N) continue;
        const int other = n_persp > 1 ? counts[(size_t)(1 - p) * N + f] : 0;
        if (n > 1 && max(n, other) > sort_limit) long_queue[atomicAdd(counters + INV_QUEUED, 1)] = p * N + f;
        if (p > 0) continue;
        const int len = n + other;
        if (len <= BWD_PART) continue;
        const int parts = (len + BWD_PART - 1) / BWD_PART;
        const int base = atomicAdd(counters + INV_PARTS, parts), q = atomicAdd(counters + INV_SPLIT, 1);
        split[3 * q + 0] = f;
        split[3 * q + 1] = base;
        split[3 * q + 2] = 0;  // (part, strip) sums done so far
        for (int i = 0; i < parts; ++i) work[base + i] = make_int2(q, i);
    }
}

__global__ void __launch_bounds__(256) k_feat_fill(const int* __restrict__ idx_stm, const int* __restrict__ idx_nstm,
                                                   const int* __restrict__ nnz, unsigned cells, unsigned A, int N,
                                                   const int* __restrict__ offsets, const int* __restrict__ ranks,
                                                   int* __restrict__ lists) {
    const int* idx = blockIdx.y ? idx_nstm : idx_stm;
    const int* off = offsets + (size_t)blockIdx.y * N;
    const int* rank = ranks + (size_t)blockIdx.y * cells;
    int* L = lists + (size_t)blockIdx.y * cells;
    for (unsigned r = blockIdx.x * 256 + threadIdx.x; r < cells; r += gridDim.x * 256) {
        const unsigned b = r / A, a = r - b * A;
        const int f = idx[r];
        if ((int)a < nnz[b] && (unsigned)f < (unsigned)N) L[off[f] + rank[r]] = (int)b;
    }
}

// The ranked scatter leaves every list in arrival order; the backward sums run in position order (deterministic results).
// Lists that fit the gradient kernel's shared memory are sorted there.  Longer ones are sorted here, one block per list: it
// marks the positions in a shared-memory bitmap and reads the set bits back in order; a list that names a position twice
// (only possible when the caller's index row repeats a feature) falls back to ranking by counting.
__global__ void __launch_bounds__(256) k_lists_sort_long(const int* __restrict__ counts, const int* __restrict__ offsets, int N,
                                                          size_t cells, int* __restrict__ lists, int* __restrict__ scratch,
                                                          const int* __restrict__ long_queue,
                                                          const int* __restrict__ long_count, int bitmap_words) {
    extern __shared__ unsigned s_bits[];  // [bitmap_words]; 0 words: always use the counting fallback
    __shared__ int s_warp[8];
    __shared__ int s_total;
    const int n_long = *long_count;
    for (int q = blockIdx.x; q < n_long; q += gridDim.x) {
        const int id = long_queue[q];
        const int p = id / N;
        const int beg = offsets[id], len = counts[id];
        int* L = lists + p * cells + beg;
        bool done = false;
        if (bitmap_words > 0) {
            for (int i = threadIdx.x; i < bitmap_words; i += blockDim.x) s_bits[i] = 0u;
            __syncthreads();
            for (int i = threadIdx.x; i < len; i += blockDim.x) {
                const int b = L[i];
                atomicOr(&s_bits[b >> 5], 1u << (b & 31));
            }
            __syncthreads();
            const int per = (bitmap_words + blockDim.x - 1) / blockDim.x;
            const int w0 = threadIdx.x * per, w1 = min(w0 + per, bitmap_words);
            int cnt = 0;
            for (int w = w0; w < w1; ++w) cnt += __popc(s_bits[w]);
            // block exclusive scan of cnt
            const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
            int incl = cnt;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                int t = __shfl_up_sync(0xffffffffu, incl, d);
                if (lane >= d) incl += t;
            }
            if (lane == 31) s_warp[wid] = incl;
            __syncthreads();
            if (threadIdx.x == 0) {
                int run = 0;
                for (int i = 0; i < 8; ++i) { int t = s_warp[i]; s_warp[i] = run; run += t; }
                s_total = run;
            }
            __syncthreads();
            if (s_total == len) {
                int pos = s_warp[wid] + incl - cnt;
                for (int w = w0; w < w1; ++w) {
                    unsigned bits = s_bits[w];
                    while (bits) {
                        const int bit = __ffs(bits) - 1;
                        bits &= bits - 1;
                        L[pos++] = (w << 5) + bit;
                    }
                }
                done = true;
            }
            __syncthreads();
        }
        if (!done) {
            int* S = scratch + p * cells + beg;
            for (int i = threadIdx.x; i < len; i += blockDim.x) S[i] = L[i];
            __syncthreads();
            for (int i = threadIdx.x; i < len; i += blockDim.x) {
                const int v = S[i];
                int r = 0;
                for (int j = 0; j < len; ++j) {
                    const int u = S[j];
                    r += (u < v) || (u == v && j < i);
                }
                L[r] = v;
            }
            __syncthreads();
        }
    }
}

// ------------------------------------------------------------------------------------------------
// backward: groups of threads own a feature row each, a thread a float4 column of it.  The row of the gradient is written
// exactly once per step (stm list first, then nstm list, each in ascending position order: the accumulation order of
// sparse_ft_backward_cpu called for stm then nstm).
//
// Bound: the gradient rows of the positions are read once per list entry, from L2 (4.0 GB at 16 384 x 1536 with 40 slots: 290
// us, 13.8 TB/s; 362 before).  What it took: strips of columns narrow enough that a strip of all rows stays in L2
// (BWD_STRIP_BYTES), the rows of a group as one stream of entries with eight 16-byte loads in flight across the ends of rows
// (lists of nine entries left half of the loads of their second round out), and two float4 columns per thread (the instructions
// per byte were the bound then: 378 to 310 us).
//
// Every warp sorts the lists of its rows into shared memory first: they are short, a few entries in a large feature space, and
// a separate pass over all rows took 27 to 30 us.
//
// Splitting: a feature that is active in very many positions (the king square of a king bucket, a pawn in hand) makes one
// group walk a list of thousands of rows; with real, skewed data such lists reach tens of thousands of entries and would
// set the kernel's run time on their own.  Rows whose lists (stm + nstm) exceed BWD_PART entries are cut into parts; every
// part of a strip is summed by its own group, ahead of the short rows, and the last one to finish adds the parts of the row
// in order.  Which group gets which part depends on timing, the sums do not.
// ------------------------------------------------------------------------------------------------
#define BWD_SORT_CELLS 256            // list cells of a warp's rows in shared memory (per perspective)
#define BWD_STRIP_BYTES (70ll << 20)
#define BWD_CELL_LAST 0x80000000  // cell flags: the row's last entry; a position of the nstm list
#define BWD_CELL_NSTM 0x40000000
#define BWD_SPLIT_BLOCKS 296          // blocks in front of the short rows' that take the parts of split rows

// Rows of a warp: with lists of a few entries a block's start costs more than the sums of eight rows (1000 positions over
// 125 388 rows of 256: 82 us with one row per warp, 66 with four).  Four rows share the sorting cells, so longer lists, which
// would have to go through k_lists_sort_long, keep one.
static inline int bwd_rows_per_warp(int B, int A, int N) { return (long long)B * A <= 16ll * N ? 4 : 1; }

template <bool DH>
static __device__ __forceinline__ float4 sum_rows(const void* __restrict__ d, const int* L, int n, int F, int c, float4 acc) {
    for (int j = 0; j < n; j += 8) {
        float4 v[8];
        // all loads of a round are in flight together; the slots behind the end add nothing
#pragma unroll
        for (int u = 0; u < 8; ++u)
            v[u] = j + u < n ? ld4<DH>(d, (size_t)L[j + u] * F + 4 * c) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int u = 0; u < 8; ++u) { acc.x += v[u].x; acc.y += v[u].y; acc.z += v[u].z; acc.w += v[u].w; }
    }
    return acc;
}

// DH: the incoming gradient rows are fp16 (summed in fp32, native_kernels.cu:1081-1140); the sums are then left in the
// rows' loss scale, which the optimizer takes out again
template <bool DH, int V>
__global__ void __launch_bounds__(256) k_ft_backward(const void* __restrict__ dft_stm, const void* __restrict__ dft_nstm,
                                                     const int* __restrict__ counts, const int* __restrict__ offsets,
                                                     const int* __restrict__ lists, size_t cells, int N, int F, int n_persp,
                                                     int strip4, int rpw, const int* __restrict__ counters,
                                                     const int2* __restrict__ work, int* split, float* partial,
                                                     float* __restrict__ grad) {
    extern __shared__ int s_mem[];  // per warp: raw cells, then sorted cells of either perspective
    __shared__ int s_off[2][32], s_len[2][32], s_beg[33], s_last[8];
    const int ths = strip4 / V;  // threads of a group: thread ct owns the float4 columns ct, ct + ths, ..
    const int groups = blockDim.x / ths, g = threadIdx.x / ths, ct = threadIdx.x - g * ths;
    const int row4 = F >> 2, c = blockIdx.y * strip4 + ct;

    if (blockIdx.x < BWD_SPLIT_BLOCKS) {
        const int n_work = counters[INV_PARTS];
        for (int w0 = blockIdx.x * groups; w0 < n_work; w0 += BWD_SPLIT_BLOCKS * groups) {
            const int w = w0 + g;
            int q = 0, f = 0, len0 = 0, len1 = 0;
            if (w < n_work) {
                const int2 wk = work[w];
                q = wk.x;
                f = split[3 * q];
                len0 = counts[f];
                len1 = n_persp > 1 ? counts[(size_t)N + f] : 0;
                const int lo = wk.y * BWD_PART, hi = min(lo + BWD_PART, len0 + len1);  // range in the concatenated lists
#pragma unroll
                for (int i = 0; i < V; ++i) {
                    const int ci = c + i * ths;
                    if (ci >= row4) break;
                    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (lo < len0) acc = sum_rows<DH>(dft_stm, lists + offsets[f] + lo, min(hi, len0) - lo, F, ci, acc);
                    if (hi > len0) {
                        const int a = max(lo - len0, 0);
                        acc = sum_rows<DH>(dft_nstm, lists + cells + offsets[(size_t)N + f] + a, hi - len0 - a, F, ci, acc);
                    }
                    reinterpret_cast<float4*>(partial)[(size_t)w * row4 + ci] = acc;
                }
                __threadfence();
            }
            __syncthreads();
            const int parts = (len0 + len1 + BWD_PART - 1) / BWD_PART;
            if (ct == 0) s_last[g] = w < n_work && atomicAdd(split + 3 * q + 2, 1) == parts * (int)gridDim.y - 1;
            __syncthreads();
            if (s_last[g]) {  // every part of every strip is there
                __threadfence();
                const float4* p4 = reinterpret_cast<const float4*>(partial) + (size_t)split[3 * q + 1] * row4;
                for (int k = ct; k < row4; k += ths) {
                    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
                    for (int i = 0; i < parts; ++i) {
                        const float4 v = __ldcg(p4 + (size_t)i * row4 + k);
                        acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
                    }
                    reinterpret_cast<float4*>(grad)[(size_t)f * row4 + k] = acc;
                }
            }
        }
        return;
    }

    const int warps = blockDim.x >> 5, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int rows = warps * rpw, r0 = (blockIdx.x - BWD_SPLIT_BLOCKS) * rows;
    const int limit = BWD_SORT_CELLS / rpw;
    if (threadIdx.x < 32) {  // at most 32 rows
        const int f = r0 + lane;
        const bool in = lane < rows && f < N;
        const int n0 = in ? counts[f] : 0, n1 = in && n_persp > 1 ? counts[(size_t)N + f] : 0;
        s_off[0][lane] = in ? offsets[f] : 0;
        s_off[1][lane] = in && n_persp > 1 ? offsets[(size_t)N + f] : 0;
        s_len[0][lane] = n0;
        s_len[1][lane] = n1;
        const int n = max(n0, n1) <= limit ? n0 + n1 : 0;
        int incl = n;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d) incl += t;
        }
        s_beg[lane + 1] = incl;
        if (lane == 0) s_beg[0] = 0;
    }
    __syncthreads();
    int* cells_s = s_mem + warps * BWD_SORT_CELLS;
    {   // the warp's lists into shared memory, then every entry to its place: the number of smaller ones before it (equal
        // ones, from a repeated feature, by index)
        int* raw = s_mem + wid * BWD_SORT_CELLS;
        for (int p = 0; p < n_persp; ++p) {
            for (int j = 0; j < rpw; ++j) {
                const int k = wid * rpw + j, n = s_len[p][k];
                if (s_beg[k + 1] == s_beg[k]) continue;
                const int* L = lists + p * cells + s_off[p][k];
                for (int i = lane; i < n; i += 32) raw[j * limit + i] = L[i];
            }
            __syncwarp();
            for (int j = 0; j < rpw; ++j) {
                const int k = wid * rpw + j, n = s_len[p][k], end = s_beg[k + 1] - 1;
                if (end < s_beg[k]) continue;
                const int* L = raw + j * limit;
                const int base = s_beg[k] + (p ? s_len[0][k] : 0);
                for (int i = lane; i < n; i += 32) {
                    const int v = L[i];
                    int r = base;
#pragma unroll 4
                    for (int m = 0; m < n; ++m) {
                        const int u = L[m];
                        r += (u < v) || (u == v && m < i);
                    }
                    cells_s[r] = v | (p ? BWD_CELL_NSTM : 0) | (r == end ? BWD_CELL_LAST : 0);
                }
            }
            __syncwarp();
        }
    }
    __syncthreads();
    if (c >= row4) return;
    float4* out = reinterpret_cast<float4*>(grad) + (size_t)r0 * row4 + c;
    const int per = (rows + groups - 1) / groups, k0 = min(g * per, rows), k1 = min(min(k0 + per, rows), N - r0);
    // rows without entries, and rows too long for shared memory
    for (int k = k0; k < k1; ++k) {
        if (s_beg[k + 1] > s_beg[k]) continue;
        const int n0 = s_len[0][k], n1 = s_len[1][k];
        if (n0 + n1 > BWD_PART) continue;  // summed in parts
#pragma unroll
        for (int i = 0; i < V; ++i) {
            float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
            acc = sum_rows<DH>(dft_stm, lists + s_off[0][k], n0, F, c + i * ths, acc);
            acc = sum_rows<DH>(dft_nstm, lists + cells + s_off[1][k], n1, F, c + i * ths, acc);
            __stcs(out + (size_t)k * row4 + i * ths, acc);
        }
    }
    // the other rows as one stream of entries, eight loads in flight across the ends of rows
    constexpr int D = 8 / V;
    const int e0 = s_beg[k0], e1 = k1 > k0 ? s_beg[k1] : e0;
    float4 v[D][V], acc[V];
    auto load = [&](int e, float4 (&x)[V]) {
        const int cell = cells_s[e];
        const void* d = cell & BWD_CELL_NSTM ? dft_nstm : dft_stm;
        const size_t at = (size_t)(cell & (BWD_CELL_NSTM - 1)) * F + 4 * c;
#pragma unroll
        for (int i = 0; i < V; ++i) x[i] = ld4<DH>(d, at + 4 * i * ths);
    };
#pragma unroll
    for (int u = 0; u < D; ++u)
        if (e0 + u < e1) load(e0 + u, v[u]);
#pragma unroll
    for (int i = 0; i < V; ++i) acc[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    int k = k0;
    for (int e = e0; e < e1; e += D) {
#pragma unroll
        for (int u = 0; u < D; ++u) {
            if (e + u >= e1) break;
#pragma unroll
            for (int i = 0; i < V; ++i) { acc[i].x += v[u][i].x; acc[i].y += v[u][i].y; acc[i].z += v[u][i].z; acc[i].w += v[u][i].w; }
            if (e + u + D < e1) load(e + u + D, v[u]);
            if (cells_s[e + u] < 0) {  // BWD_CELL_LAST
                while (s_beg[k + 1] <= e + u) ++k;  // past rows without entries here
#pragma unroll
                for (int i = 0; i < V; ++i) {
                    __stcs(out + (size_t)k * row4 + i * ths, acc[i]);  // not read again in this launch: L2 is the input's
                    acc[i] = make_float4(0.f, 0.f, 0.f, 0.f);
                }
            }
        }
    }
}

int launch_inverse_index(cudaStream_t s, const int* idx_stm, const int* idx_nstm, const int* nnz, int B, int A, int N, int n_persp,
                         int* counts, int* offsets, int* lists, int* plan) {
    if (B <= 0) return 0;
    const unsigned cells = (unsigned)B * (unsigned)A;
    int* counters = counts + (size_t)2 * N;
    int* long_queue = counters + INV_COUNTERS;
    int* scratch = lists + (size_t)2 * cells;  // the ranks, then the long sort's copies
    int2* work = reinterpret_cast<int2*>(plan);
    int* split = plan + 2 * (size_t)ft_backward_max_work(B, A, n_persp);
    cudaMemsetAsync(counts, 0, sizeof(int) * ((size_t)2 * N + INV_COUNTERS), s);
    const dim3 grid((unsigned)min(ceil_div(cells, 256), sm_count() * 16), n_persp);
    k_feat_count<<<grid, 256, 0, s>>>(idx_stm, idx_nstm, nnz, cells, A, N, counts, scratch);
    k_feat_scan<<<dim3(ceil_div(N, SCAN_CELLS), n_persp), 1024, 0, s>>>(counts, N, n_persp, BWD_SORT_CELLS / bwd_rows_per_warp(B, A, N),
                                                                        offsets, counters, long_queue, work, split);
    k_feat_fill<<<grid, 256, 0, s>>>(idx_stm, idx_nstm, nnz, cells, A, N, offsets, scratch, lists);
    int words = (B + 31) / 32;
    if ((size_t)words * 4 > 160 * 1024) words = 0;
    // per device and cheap: set before every launch (a process may drive several GPUs)
    cudaFuncSetAttribute(k_lists_sort_long, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024);
    k_lists_sort_long<<<sm_count() * 4, 256, (size_t)words * 4, s>>>(counts, offsets, N, cells, lists, scratch, long_queue,
                                                              counters + INV_QUEUED, words);
    return 4;
}

int ft_backward_max_work(int B, int A, int n_persp) { return 2 * (int)(((long long)n_persp * B * A) / BWD_PART) + 2; }

int launch_ft_backward_split(cudaStream_t s, const void* dft_stm, const void* dft_nstm, const int* counts, const int* offsets,
                             const int* lists, int B, int A, int N, int F, int n_persp, int* plan, float* partial, float* grad,
                             int dft_half) {
    const int2* work = reinterpret_cast<const int2*>(plan);
    int* split = plan + 2 * (size_t)ft_backward_max_work(B, A, n_persp);
    // The widest strips of whole 128-column pieces that keep the input in L2 and a group within a block; two pieces are not
    // cut.  Two float4 columns per thread where the strips allow it: half the instructions per byte.
    const int pieces = F / 128;
    int ny = 0, per, v;
    do {
        per = ceil_div(pieces, ++ny);
        v = per % 2 == 0 && pieces % per == 0 ? 2 : 1;
    } while (per / v > 8 || (per > 2 && (long long)n_persp * B * per * (dft_half ? 256 : 512) > BWD_STRIP_BYTES));
    ny = ceil_div(pieces, per);
    const int strip4 = 32 * per, ths = strip4 / v, threads = ths * (ths < 256 ? 256 / ths : 1);
    const int warps = threads / 32, rpw = bwd_rows_per_warp(B, A, N);
    const dim3 grid(BWD_SPLIT_BLOCKS + ceil_div(N, warps * rpw), ny);
    const size_t smem = sizeof(int) * BWD_SORT_CELLS * warps * (1 + n_persp);
    const size_t cells = (size_t)B * A;
    auto* kernel = dft_half ? (v == 2 ? k_ft_backward<true, 2> : k_ft_backward<true, 1>)
                            : (v == 2 ? k_ft_backward<false, 2> : k_ft_backward<false, 1>);
    kernel<<<grid, threads, smem, s>>>(dft_stm, dft_nstm, counts, offsets, lists, cells, N, F, n_persp, strip4, rpw,
                                       counts + (size_t)2 * N, work, split, partial, grad);
    return 1;
}

// ft_reduce_virtual_grad (sparse/ft_factorize.rs:109-121): grad[N + v] = sum over king buckets of grad[kb*pi + v]
__global__ void k_ft_reduce_virtual(float* __restrict__ grad, int N, int pi, int F) {
    const int row4 = F >> 2;
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= (long long)pi * row4) return;
    const int v = (int)(i / row4), c = (int)(i - (long long)v * row4);
    const float4* g4 = reinterpret_cast<const float4*>(grad);
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int f = v; f < N; f += pi) {
        const float4 x = g4[(size_t)f * row4 + c];
        acc.x += x.x; acc.y += x.y; acc.z += x.z; acc.w += x.w;
    }
    reinterpret_cast<float4*>(grad)[(size_t)(N + v) * row4 + c] = acc;
}

int launch_ft_reduce_virtual(cudaStream_t s, float* grad, int N, int pi, int F) {
    const long long n = (long long)pi * (F / 4);
    k_ft_reduce_virtual<<<(int)((n + 255) / 256), 256, 0, s>>>(grad, N, pi, F);
    return 1;
}

// ft_fold_virtual (sparse/ft_factorize.rs:78-99): comb[f] = w[f] + w[N + f % pi]; HC: rounded to fp16
// (ft_fold_virtual_f16, native_kernels.cu:262-318)
template <bool HC>
__global__ void k_ft_fold(const float* __restrict__ w, void* __restrict__ comb, int N, int pi, int F) {
    const int row4 = F >> 2;
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= (long long)N * row4) return;
    const int f = (int)(i / row4), c = (int)(i - (long long)f * row4);
    const float4* w4 = reinterpret_cast<const float4*>(w);
    const float4 a = w4[i];
    const float4 b = w4[(size_t)(N + f % pi) * row4 + c];
    const float4 v = make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
    if (HC) static_cast<uint2*>(comb)[i] = make_uint2(pack_h2(v.x, v.y), pack_h2(v.z, v.w));
    else static_cast<float4*>(comb)[i] = v;
}

int launch_ft_fold(cudaStream_t s, const float* w, void* comb, int N, int pi, int F, int half_comb) {
    const long long n = (long long)N * (F / 4);
    if (half_comb) k_ft_fold<true><<<(int)((n + 255) / 256), 256, 0, s>>>(w, comb, N, pi, F);
    else k_ft_fold<false><<<(int)((n + 255) / 256), 256, 0, s>>>(w, comb, N, pi, F);
    return 1;
}

// cast_f32_to_f16 (native_kernels.cu:648): the fp16 mirror of an fp32 table
__global__ void k_cast_half(const float4* __restrict__ src, uint2* __restrict__ dst, long long n4) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n4; i += (long long)gridDim.x * blockDim.x) {
        const float4 v = src[i];
        dst[i] = make_uint2(pack_h2(v.x, v.y), pack_h2(v.z, v.w));
    }
}

int launch_cast_half(cudaStream_t s, const float* src, void* dst, int64_t n) {
    const long long n4 = n / 4;
    long long blocks = (n4 + 255) / 256;
    blocks = blocks < 16 * sm_count() ? blocks : 16 * sm_count();
    if (blocks < 1) blocks = 1;
    k_cast_half<<<(int)blocks, 256, 0, s>>>(reinterpret_cast<const float4*>(src), static_cast<uint2*>(dst), n4);
    return 1;
}
