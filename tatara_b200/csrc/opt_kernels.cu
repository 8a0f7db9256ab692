// Optimizer kernels: the RAdam / Ranger / AdamW update with weight clamp (radam_step,
// native_kernels.cu:1291; pointwise/radam_step.rs:116-156) and the Ranger look-ahead interpolation
// (native_kernels.cu:1842; pointwise/ranger_step.rs:52-59), fused so that every parameter and moment
// crosses HBM once per step.  The gradient is only read: every gradient buffer is fully rewritten by
// the next backward pass, so the reference's grad = 0 store is not needed.
#include "radam.cuh"

// plain streaming update of one large group (n multiple of 4); mirror: optional fp16 copy of the updated weights
// (radam_step_fp16_mirror / radam_step_f16state_mirror + ranger_lookahead_lerp_fp16_mirror, native_kernels.cu:1183-1290)
template <bool HS>
__global__ void __launch_bounds__(256) k_radam(float4* __restrict__ w, void* __restrict__ m, void* __restrict__ v,
                                                const float4* __restrict__ g, float4* __restrict__ slow, uint2* __restrict__ mirror,
                                                long long n4, OptScalars sc) {
    const float rate = radam_rate(sc);
    const float decay_mul = radam_decay(sc, rate);
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n4; i += (long long)gridDim.x * blockDim.x) {
        float4 mi = load_moment<HS>(m, i, 1.0f / TB_FT_OPT_M_SCALE, false), vi = load_moment<HS>(v, i, 1.0f / TB_FT_OPT_V_SCALE, false);
        float4 p = radam_four<RADAM_TABLE>(w[i], mi, vi, scale4(g[i], sc.grad_scale), sc, rate, decay_mul);
        store_moment<HS>(m, i, mi, TB_FT_OPT_M_SCALE, true, false);
        store_moment<HS>(v, i, vi, TB_FT_OPT_V_SCALE, false, false);
        if (sc.lerp) {
            p = lerp_four(p, slow[i], sc.alpha);
            slow[i] = p;
        }
        w[i] = p;
        if (mirror) mirror[i] = pack_h4(p);
    }
}

int launch_radam(cudaStream_t s, float* w, void* m, void* v, const float* g, float* slow, int64_t n, OptScalars sc, int half_state,
                 void* mirror) {
    const long long n4 = n / 4;
    long long blocks = (n4 + 255) / 256;
    const long long most = 32 * sm_count();
    if (blocks > most) blocks = most;
    if (blocks < 1) blocks = 1;
    if (half_state)
        k_radam<true><<<(int)blocks, 256, 0, s>>>(reinterpret_cast<float4*>(w), m, v, reinterpret_cast<const float4*>(g),
                                                  reinterpret_cast<float4*>(slow), static_cast<uint2*>(mirror), n4, sc);
    else
        k_radam<false><<<(int)blocks, 256, 0, s>>>(reinterpret_cast<float4*>(w), m, v, reinterpret_cast<const float4*>(g),
                                                   reinterpret_cast<float4*>(slow), static_cast<uint2*>(mirror), n4, sc);
    return 1;
}

// all small groups in one launch: grid (groups, blocks)
__global__ void __launch_bounds__(256) k_radam_small(const __grid_constant__ SmallGroups groups, OptScalars sc) {
    const SmallGroup gr = groups.g[blockIdx.x];
    sc.lr = gr.lr;
    sc.decay = gr.decay;
    sc.min_w = gr.min_w;
    sc.max_w = gr.max_w;
    const float rate = radam_rate(sc);
    const float decay_mul = radam_decay(sc, rate);
    for (int i = blockIdx.y * blockDim.x + threadIdx.x; i < gr.n; i += gridDim.y * blockDim.x) {
        float mi = gr.m[i], vi = gr.v[i];
        float p = radam_one<RADAM_SMALL>(gr.w[i], mi, vi, gr.grad[i], sc, rate, decay_mul);
        gr.m[i] = mi;
        gr.v[i] = vi;
        if (sc.lerp) {
            p = sc.alpha * p + (1.0f - sc.alpha) * gr.slow[i];
            gr.slow[i] = p;
        }
        gr.w[i] = p;
    }
}

int launch_radam_small(cudaStream_t s, const SmallGroups& groups, int max_n, OptScalars sc) {
    int by = ceil_div(max_n, 256 * 4);
    if (by < 1) by = 1;
    if (by > 512) by = 512;
    k_radam_small<<<dim3(groups.n, by), 256, 0, s>>>(groups, sc);
    return 1;
}

// asynchronous copy of 8 or 16 bytes global -> shared (both aligned to that)
template <int BYTES>
static __device__ __forceinline__ void ok_cp(void* dst_shared, const void* src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst_shared);
    if (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
}

// ------------------------------------------------------------------------------------------------
// Factorised FT table (N = KB * pi real rows + pi virtual rows).  A block owns 32 adjacent float4 columns of one virtual row
// vr, its warps share that row's KB real rows kb*pi + vr, up to FACT_ROWS neighbours each:
//   - the rows' gradients go into shared memory, where 128 threads add them up in kb order, one chain per column: the virtual
//     row's gradient (ft_reduce_virtual_grad, sparse/ft_factorize.rs:109-121);
//   - every warp updates its rows, the first one also the virtual row N + vr;
//   - comb[kb*pi + v] = w[kb*pi + v] + w[N + v] (ft_fold_virtual, sparse/ft_factorize.rs:78-99), the updated real rows kept in
//     shared memory, where their gradients were.
// Replaces radam_step on N_t*F elements + ft_reduce_virtual_grad + ranger_lookahead_lerp + ft_fold_virtual.
// HBM-bound.  With a thread per column walking all the rows twice, the second walk found them gone from L2 (122 MB of rows
// in flight): 4.2 GB moved instead of the 3.8 needed.  Warps side by side also make enough loads in flight where the table
// is narrow.  F = 1536 / 768 / 256, 45 king buckets, fp32: 730 / 373 / 140 us with the walks, 626 / 319 / 123 now (0.93 of
// the measured HBM rate at 1536); fp16 moments and table at 1536: 566, now 499.  (Rows in registers: 667.  No folded table,
// the forward adding the two rows as it loads a strip: 566 here, but 190 more there.  Every warp adding up its own rows and
// the warps' sums after that: 637 / 325 / 122 and 492, another order.  The chain by a warp that reads the rows itself: 970.)
#define FACT_ROWS 9   // rows of a warp: 45 and 81 king buckets are 5 and 9 full warps
#define FACT_BATCH 3  // of these, loaded together
// HS: fp16 moments; HC: fp16 folded table.  The real rows' gradients are multiplied by sc.grad_scale on load; the virtual
// row's gradient cell receives the sum of the scaled values (its true gradient).
template <int MAX_WARPS, int MIN_BLOCKS, bool HS, bool HC>
__global__ void __launch_bounds__(32 * MAX_WARPS, MIN_BLOCKS) k_radam_factorized(float4* __restrict__ w, void* __restrict__ m, void* __restrict__ v,
                                                            float4* __restrict__ g, float4* __restrict__ slow,
                                                            void* __restrict__ comb, int N, int pi, int row4, OptScalars sc) {
    __shared__ float4 s_virt[32];  // the virtual row: its gradient, then the updated weights
    __shared__ float4 s_row[FACT_ROWS][32 * MAX_WARPS];  // the real rows: likewise
    __shared__ float4 s_vw[32], s_vm[32], s_vv[32];  // weights and moments (as stored) of the virtual row
    const float inv_ms = 1.0f / TB_FT_OPT_M_SCALE, inv_vs = 1.0f / TB_FT_OPT_V_SCALE;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const size_t plane = (size_t)pi * row4;  // float4 of one king bucket
    const size_t cell = (size_t)blockIdx.x * 32 + lane;  // a row is a multiple of 32 float4 long
    const int KB = N / pi;
    const int kb0 = warp * FACT_ROWS;
    const float rate = radam_rate(sc);
    const float decay_mul = radam_decay(sc, rate);
#pragma unroll
    for (int u = 0; u < FACT_ROWS; ++u)
        if (kb0 + u < KB) ok_cp<16>(&s_row[u][threadIdx.x], g + (size_t)(kb0 + u) * plane + cell);
    const size_t iv = (size_t)KB * plane + cell;
    constexpr int MSZ = HS ? 8 : 16;  // bytes of four moments
    if (warp == 0) {
        ok_cp<16>(&s_vw[lane], w + iv);
        ok_cp<MSZ>(reinterpret_cast<char*>(s_vm) + lane * MSZ, static_cast<const char*>(m) + iv * MSZ);
        ok_cp<MSZ>(reinterpret_cast<char*>(s_vv) + lane * MSZ, static_cast<const char*>(v) + iv * MSZ);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    float4 p[FACT_BATCH], mi[FACT_BATCH], vi[FACT_BATCH];
    auto load = [&](int b) {  // everything streams through once: evict-first
#pragma unroll
        for (int u = 0; u < FACT_BATCH; ++u) {
            const size_t i = (size_t)min(kb0 + b + u, KB - 1) * plane + cell;  // past the end: the last row, dropped below
            p[u] = __ldcs(w + i);
            mi[u] = load_moment<HS>(m, i, inv_ms, true);
            vi[u] = load_moment<HS>(v, i, inv_vs, true);
        }
    };
    load(0);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    for (int c = threadIdx.x; c < 128; c += blockDim.x) {
        const float* col = reinterpret_cast<const float*>(s_row) + c;
        float sum = 0.f;
        int kb = 0;
        for (int q = 0; q < warps; ++q)
#pragma unroll
            for (int u = 0; u < FACT_ROWS; ++u, ++kb) {
                if (kb >= KB) break;
                float x = col[(u * 32 * MAX_WARPS + 32 * q) * 4];
                if (HC) x = __fmul_rn(x, sc.grad_scale);  // loss-scaled sums exist only next to an fp16 table
                sum += x;
            }
        reinterpret_cast<float*>(s_virt)[c] = sum;
    }
    __syncthreads();
    if (warp == 0) {
        const float4 gsum = s_virt[lane];
        g[iv] = gsum;
        float4 mv = load_moment<HS>(s_vm, lane, inv_ms, false), vv = load_moment<HS>(s_vv, lane, inv_vs, false);
        float4 pv = radam_four<RADAM_FACT, RADAM_FACT_LAST>(s_vw[lane], mv, vv, gsum, sc, rate, decay_mul);
        store_moment<HS>(m, iv, mv, TB_FT_OPT_M_SCALE, true, false);
        store_moment<HS>(v, iv, vv, TB_FT_OPT_V_SCALE, false, false);
        if (sc.lerp) {
            pv = lerp_four(pv, slow[iv], sc.alpha);
            slow[iv] = pv;
        }
        w[iv] = pv;
        s_virt[lane] = pv;
    }
#pragma unroll 1
    for (int b = 0; b < FACT_ROWS; b += FACT_BATCH) {
#pragma unroll
        for (int u = 0; u < FACT_BATCH; ++u) {
            if (kb0 + b + u >= KB) break;
            const size_t i = (size_t)(kb0 + b + u) * plane + cell;
            float4 gi = s_row[b + u][threadIdx.x];
            if (HC) gi = scale4(gi, sc.grad_scale);
            float4 q = radam_four<RADAM_FACT>(p[u], mi[u], vi[u], gi, sc, rate, decay_mul);
            store_moment<HS>(m, i, mi[u], TB_FT_OPT_M_SCALE, true, true);
            store_moment<HS>(v, i, vi[u], TB_FT_OPT_V_SCALE, false, true);
            if (sc.lerp) {
                q = lerp_four(q, __ldcs(slow + i), sc.alpha);
                __stcs(slow + i, q);
            }
            __stcs(w + i, q);
            s_row[b + u][threadIdx.x] = q;
        }
        if (b + FACT_BATCH < FACT_ROWS) load(b + FACT_BATCH);
    }
    __syncthreads();
    const float4 pv = s_virt[lane];
#pragma unroll
    for (int u = 0; u < FACT_ROWS; ++u) {
        if (kb0 + u >= KB) break;
        const size_t i = (size_t)(kb0 + u) * plane + cell;
        const float4 p = s_row[u][threadIdx.x];
        const float4 f = make_float4(p.x + pv.x, p.y + pv.y, p.z + pv.z, p.w + pv.w);
        if (HC) __stcs(static_cast<uint2*>(comb) + i, pack_h4(f));
        else __stcs(static_cast<float4*>(comb) + i, f);
    }
}

// The same work in two kinds of launches, for the data-parallel pipeline in which the gradient rows arrive king bucket
// range by king bucket range: k_radam_factorized_rows updates the real rows of the buckets [kb0, kb1) and carries the
// running gradient sum of every virtual row through that row's gradient cell (ranges must be given in ascending
// order, so the sum is added up in the order of the fused kernel), k_radam_factorized_fold then updates the virtual
// rows and writes the folded table.  Results are bit-identical to the fused kernel.
template <bool HS, bool GS>
__global__ void __launch_bounds__(1024) k_radam_factorized_rows(float4* __restrict__ w, void* __restrict__ m, void* __restrict__ v,
                                                                 float4* __restrict__ g, float4* __restrict__ slow, int N, int pi,
                                                                 int row4, int kb0, int kb1, OptScalars sc) {
    const int vr = blockIdx.x;
    const int c = threadIdx.x;
    const float rate = radam_rate(sc);
    const float decay_mul = radam_decay(sc, rate);
    const float inv_ms = 1.0f / TB_FT_OPT_M_SCALE, inv_vs = 1.0f / TB_FT_OPT_V_SCALE;
    const size_t iv = (size_t)(N + vr) * row4 + c;
    float4 gsum = kb0 == 0 ? make_float4(0.f, 0.f, 0.f, 0.f) : g[iv];
#pragma unroll 4
    for (int kb = kb0; kb < kb1; ++kb) {
        const size_t i = (size_t)(kb * pi + vr) * row4 + c;
        float4 gi = __ldcs(g + i);
        if (GS) gi = scale4(gi, sc.grad_scale);
        float4 mi = load_moment<HS>(m, i, inv_ms, true), vi = load_moment<HS>(v, i, inv_vs, true);
        float4 p = radam_four<RADAM_FACT>(w[i], mi, vi, gi, sc, rate, decay_mul);
        store_moment<HS>(m, i, mi, TB_FT_OPT_M_SCALE, true, true);
        store_moment<HS>(v, i, vi, TB_FT_OPT_V_SCALE, false, true);
        if (sc.lerp) {
            p = lerp_four(p, __ldcs(slow + i), sc.alpha);
            __stcs(slow + i, p);
        }
        w[i] = p;
        gsum.x += gi.x; gsum.y += gi.y; gsum.z += gi.z; gsum.w += gi.w;
    }
    g[iv] = gsum;
}

template <bool HS, bool HC>
__global__ void __launch_bounds__(1024) k_radam_factorized_fold(float4* __restrict__ w, void* __restrict__ m, void* __restrict__ v,
                                                                 float4* __restrict__ g, float4* __restrict__ slow,
                                                                 void* __restrict__ comb, int N, int pi, int row4, OptScalars sc) {
    const int vr = blockIdx.x;
    const int c = threadIdx.x;
    const float rate = radam_rate(sc);
    const float decay_mul = radam_decay(sc, rate);
    const int KB = N / pi;
    const size_t iv = (size_t)(N + vr) * row4 + c;
    float4 mv = load_moment<HS>(m, iv, 1.0f / TB_FT_OPT_M_SCALE, false), vv = load_moment<HS>(v, iv, 1.0f / TB_FT_OPT_V_SCALE, false);
    float4 pv = radam_four<RADAM_FACT, RADAM_FACT_LAST>(w[iv], mv, vv, g[iv], sc, rate, decay_mul);
    store_moment<HS>(m, iv, mv, TB_FT_OPT_M_SCALE, true, false);
    store_moment<HS>(v, iv, vv, TB_FT_OPT_V_SCALE, false, false);
    if (sc.lerp) {
        pv = lerp_four(pv, slow[iv], sc.alpha);
        slow[iv] = pv;
    }
    w[iv] = pv;
#pragma unroll 4
    for (int kb = 0; kb < KB; ++kb) {
        const size_t i = (size_t)(kb * pi + vr) * row4 + c;
        const float4 p = __ldcs(w + i);
        const float4 f = make_float4(p.x + pv.x, p.y + pv.y, p.z + pv.z, p.w + pv.w);
        if (HC) __stcs(static_cast<uint2*>(comb) + i, pack_h4(f));
        else __stcs(static_cast<float4*>(comb) + i, f);
    }
}

int launch_radam_factorized_rows(cudaStream_t s, float* w, void* m, void* v, float* g, float* slow, int N, int pi, int F, int kb0,
                                 int kb1, OptScalars sc, int half_state) {
    float4 *w4 = reinterpret_cast<float4*>(w), *g4 = reinterpret_cast<float4*>(g), *s4 = reinterpret_cast<float4*>(slow);
    const bool gs = sc.grad_scale != 1.0f;
#define ROWS(HS, GS) k_radam_factorized_rows<HS, GS><<<pi, F / 4, 0, s>>>(w4, m, v, g4, s4, N, pi, F / 4, kb0, kb1, sc)
    if (half_state) { if (gs) ROWS(true, true); else ROWS(true, false); }
    else { if (gs) ROWS(false, true); else ROWS(false, false); }
#undef ROWS
    return 1;
}

int launch_radam_factorized_fold(cudaStream_t s, float* w, void* m, void* v, float* g, float* slow, void* comb, int N, int pi,
                                 int F, OptScalars sc, int half_state, int half_comb) {
    float4 *w4 = reinterpret_cast<float4*>(w), *g4 = reinterpret_cast<float4*>(g), *s4 = reinterpret_cast<float4*>(slow);
#define FOLD(HS, HC) k_radam_factorized_fold<HS, HC><<<pi, F / 4, 0, s>>>(w4, m, v, g4, s4, comb, N, pi, F / 4, sc)
    if (half_state) { if (half_comb) FOLD(true, true); else FOLD(true, false); }
    else { if (half_comb) FOLD(false, true); else FOLD(false, false); }
#undef FOLD
    return 1;
}

int launch_radam_factorized(cudaStream_t s, float* w, void* m, void* v, float* g, float* slow, void* comb, int N,
                            int pi, int F, OptScalars sc, int half_state, int half_comb) {
    float4 *w4 = reinterpret_cast<float4*>(w), *g4 = reinterpret_cast<float4*>(g), *s4 = reinterpret_cast<float4*>(slow);
    const int KB = N / pi, warps = ceil_div(KB, FACT_ROWS), blocks = (int)((long long)pi * (F / 4) / 32);
#define FUSED(MW, MB, HS, HC) k_radam_factorized<MW, MB, HS, HC><<<blocks, 32 * warps, 0, s>>>(w4, m, v, g4, s4, comb, N, pi, F / 4, sc)
#define FUSED_H(MW, MB, MBH)                                                                                                   \
    do {                                                                                                                       \
        if (half_state) { if (half_comb) FUSED(MW, MBH, true, true); else FUSED(MW, MBH, true, false); }                       \
        else { if (half_comb) FUSED(MW, MB, false, true); else FUSED(MW, MB, false, false); }                                  \
    } while (0)
    // blocks per SM, measured with the sums in registers (F = 1536, fp32 / fp16 moments): 5 blocks 636 / 506 us, 6 641 / 490, 8 with one row at
    // a time 800 / 568
    if (warps <= 5) FUSED_H(5, 5, 6);
    else if (warps <= 9) FUSED_H(9, 3, 3);
    else return launch_radam_factorized_rows(s, w, m, v, g, slow, N, pi, F, 0, KB, sc, half_state) +
                launch_radam_factorized_fold(s, w, m, v, g, slow, comb, N, pi, F, sc, half_state, half_comb);
#undef FUSED_H
#undef FUSED
    return 1;
}
