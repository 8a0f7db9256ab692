// The hidden layers behind L1 in one kernel: L1 activation .. L2 .. L3 .. loss, back to the L1 output, and the block's share of
// the weight gradients of L2, L3 and the biases (trainer_layerstack.rs:2530-2717 forward, :2976-3325 backward;
// trainer_simple.rs:1281-1508, :1560-1765; weight gradients dense_mm_bucket.rs:112-161).  For l1 = 8, 16, 32 and l2 = 16, 32;
// dense_kernels.cu has the kernels for other sizes.
//
// The order of the sums is part of the results, and the weight gradients' decides the shape: the positions of a bucket, in bucket
// order, are cut into 64 equal runs (Simple: all positions into 128), a run is one chain, and the runs are added by a tree
// (k_tail_wgrad_final).  A block owns a run and takes T of its positions at a time, a thread one of them; the gradients stay in
// registers from round to round.  The bucket's weights sit in shared memory and reach the threads as broadcasts, the position's
// vectors stay in registers; for the weight gradients the threads put them side by side in shared memory and then own cells of
// the gradient instead.  What bounds it is the latency of a block; the only large traffic is the L1 rows in and out.
// Tail and sums, 65 536 positions of a LayerStack net with l1 = 16 / of a Simple net / 1024 of a LayerStack net: 42 + 8, 46 + 8,
// 23 + 8 us.  A warp per position with every bucket's weights in each block, and the weight gradients in a kernel of their own that
// read the vectors back from memory, in the same order: 69 + 74, 65 + 92, 23 + 29; blocks of 128 positions with the weight
// gradients summed block by block, another order: 50 + 13, 41 + 14, 20 + 7.
#include "common.cuh"
#include "loss.cuh"

namespace {

// ARCH: 0 LayerStack, 1 Simple CReLU (and Pairwise), 2 Simple SCReLU; T: positions of a round, threads of a block
template <int ARCH, int L1, int L2, int T>
struct TailShape {
    static constexpr int L1E = L1 - 1;
    static constexpr int NIN = ARCH == 0 ? 2 * L1E : L1;  // inputs of L2
    static constexpr int NP = (NIN + 3) / 4 * 4;          // padded
    static constexpr int LDV = NP + 4, LDU = L2 + 4, LDD = L1 + 4;  // row strides: a quarter warp's 16-byte rows hit all banks
    static constexpr int W_FLOATS = L2 * NP + 2 * L2;
    static constexpr int STAGE = T * (LDV + 2 * LDU + LDD + 1);
    static constexpr int NW = NIN * L2;
    static constexpr int NB = 2 * L2 + 1 + L1;  // biases of L2, weights of L3, bias of L3, biases of L1
    static constexpr int CELLS = NW + NB;
};

template <int ARCH>
__device__ __forceinline__ float tail_act(float a) { return ARCH == 2 ? a * a : a; }  // of the clipped value
// derivative of the activation times up, from the clipped value (strictly inside (0, 1) exactly where the unclipped one is)
template <int ARCH>
__device__ __forceinline__ float tail_act_grad(float a, float up) {
    if (ARCH == 2) return up * ((a > 0.f && a < 1.0f) ? 2.0f * a : 0.f);
    return (a > 0.f && a < 1.0f) ? up : 0.f;
}

}  // namespace

template <int ARCH, int L1, int L2, int T>
__global__ void __launch_bounds__(T) k_tail(const float* __restrict__ l1_rows, const int* __restrict__ order,
                                            const int* __restrict__ seg_start, int split, const float* __restrict__ score,
                                            const float* __restrict__ wdl, const float* __restrict__ l2_w,
                                            const float* __restrict__ l2_b, const float* __restrict__ l3_w,
                                            const float* __restrict__ l3_b, LossParams lp, int nb,
                                            float* __restrict__ net_output, float* __restrict__ dy_out,
                                            float* __restrict__ dl1_rows, float* __restrict__ partials,
                                            double* __restrict__ loss_partials, int backward) {
    typedef TailShape<ARCH, L1, L2, T> S;
    constexpr int NIN = S::NIN, NP = S::NP, L1E = S::L1E;
    extern __shared__ __align__(16) float s_dyn[];
    float* s_w = s_dyn;                    // [L2][NP]
    float* s_b2 = s_w + L2 * NP;           // [L2]
    float* s_w3 = s_b2 + L2;               // [L2]
    float* s_v = s_dyn + S::W_FLOATS;      // [T][LDV] inputs of L2
    float* s_u = s_v + T * S::LDV;         // [T][LDU] gradient of L2's outputs
    float* s_a = s_u + T * S::LDU;         // [T][LDU] L2's activations
    float* s_d = s_a + T * S::LDU;         // [T][LDD] gradient of the L1 outputs
    float* s_y = s_d + T * S::LDD;         // [T] gradient of the output
    const int tid = threadIdx.x;
    const int g = blockIdx.x / split, sp = blockIdx.x - g * split;
    const int seg = seg_start[g], len = seg_start[g + 1] - seg, per = (len + split - 1) / split;
    const int beg = seg + min(sp * per, len), end = seg + min((sp + 1) * per, len);
    float* part = partials + (size_t)blockIdx.x * S::CELLS;
    if (beg >= end) {  // nothing here: the sums over the blocks read every row
        if (tid == 0) loss_partials[blockIdx.x] = 0.0;
        if (backward)
            for (int c = tid; c < S::CELLS; c += T) part[c] = 0.f;
        return;
    }
    const bool live = ARCH != 0 || g < nb;  // positions with a bucket id out of range have no L2 and L3
    if (live) {
        const float* w2 = l2_w + (ARCH == 0 ? (size_t)g * S::NW : 0);
        // few threads: many loads in flight each (one by one they took 5 us)
#pragma unroll 16
        for (int e = tid; e < L2 * NP; e += T) {
            const int o = e / NP, i = e % NP;
            s_w[e] = i < NIN ? (ARCH == 0 ? w2[o * NIN + i] : w2[i * L2 + o]) : 0.f;
        }
        if (tid < L2) {  // L2 <= 32 <= T
            s_b2[tid] = l2_b[(ARCH == 0 ? g * L2 : 0) + tid];
            s_w3[tid] = l3_w[(ARCH == 0 ? g * L2 : 0) + tid];
        }
    }
    const float b3 = live ? l3_b[ARCH == 0 ? g : 0] : 0.f;
    // the run's sums: four outputs and IT inputs of the L2 weights, and of the other cells every T-th
    constexpr int OQ = L2 / 4, G = T / OQ, IT = (NP + G - 1) / G, NS = (S::NB + T - 1) / T;
    const int o0 = 4 * (tid % OQ), i0 = IT * (tid / OQ);
    float acc[4][IT], other[NS];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < IT; ++b) acc[a][b] = 0.f;
#pragma unroll
    for (int j = 0; j < NS; ++j) other[j] = 0.f;
    double e2 = 0.0;
    for (int r0 = beg; r0 < end; r0 += T) {
        const int n = min(T, end - r0);
        const int pos = tid < n ? order[r0 + tid] : -1;
        const float4* row = reinterpret_cast<const float4*>(l1_rows + (size_t)(pos < 0 ? 0 : pos) * L1);
        float in[NP];  // the clipped inputs of L2
        float skip = 0.f;
#pragma unroll
        for (int i = 0; i < NP; ++i) in[i] = 0.f;
#pragma unroll
        for (int q = 0; q < L1 / 4; ++q) {
            const float4 x = pos >= 0 ? row[q] : make_float4(0.f, 0.f, 0.f, 0.f);
            const float xv[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int i = 4 * q + e;
                if (ARCH != 0) in[i] = crelu01(xv[e]);
                else if (i < L1E) {
                    in[i] = crelu01(xv[e] * xv[e] * L1_SQR_SCALE);
                    in[L1E + i] = crelu01(xv[e]);
                } else skip = xv[e];
            }
        }
        const float sc = pos >= 0 ? score[pos] : 0.f, wd = pos >= 0 ? wdl[pos] : 0.f;
        __syncthreads();  // the weights; from the second round on: the sums have read the last round's vectors
        float a2[L2];  // L2's clipped outputs
        float out = skip;
        if (live) {
            // L3: the products are added by a tree (LayerStack with l1 = 32: one chain from the bias)
            constexpr bool TREE = ARCH != 0 || L1 <= 16;
            float l3 = b3, term[32];
#pragma unroll
            for (int o = 0; o < 32; ++o) term[o] = 0.f;
#pragma unroll
            for (int o = 0; o < L2; ++o) {
                // weights of two outputs at a time: the compiler otherwise brings those of all in first, far beyond the registers
                if (o % 2 == 0) asm volatile("" ::: "memory");
                float sum = s_b2[o];
#pragma unroll
                for (int i4 = 0; i4 < NP / 4; ++i4) {
                    const float4 w = *reinterpret_cast<const float4*>(s_w + o * NP + 4 * i4);
                    const float* x = in + 4 * i4;
                    sum += tail_act<ARCH>(x[0]) * w.x; sum += tail_act<ARCH>(x[1]) * w.y;
                    sum += tail_act<ARCH>(x[2]) * w.z; sum += tail_act<ARCH>(x[3]) * w.w;
                }
                a2[o] = crelu01(sum);
                if (TREE) term[o] = __fmul_rn(tail_act<ARCH>(a2[o]), s_w3[o]);
                else l3 += tail_act<ARCH>(a2[o]) * s_w3[o];
            }
            if (TREE) {
#pragma unroll
                for (int d = 16; d > 0; d >>= 1)
#pragma unroll
                    for (int o = 0; o < d; ++o) term[o] = __fadd_rn(term[o], term[o + d]);
                l3 = __fadd_rn(b3, term[0]);
            }
            out = ARCH == 0 ? l3 + skip : l3;
        } else {
#pragma unroll
            for (int o = 0; o < L2; ++o) a2[o] = 0.f;
        }
        float dy = 0.f;
        if (pos >= 0) {
            e2 += loss_point(lp, out, sc, wd, &dy);
            net_output[pos] = out;
            dy_out[pos] = dy;
        }
        if (!backward) continue;

        // back to the L1 output; the position's vectors go into shared memory on the way (zeros past the block's positions)
        float dp[NP];
#pragma unroll
        for (int i = 0; i < NP; ++i) dp[i] = 0.f;
#pragma unroll
        for (int o4 = 0; o4 < L2; o4 += 4) {
            asm volatile("" ::: "memory");
            float d[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int o = o4 + e;
                d[e] = live ? tail_act_grad<ARCH>(a2[o], dy * s_w3[o]) : 0.f;
                if (live) {
#pragma unroll
                    for (int i4 = 0; i4 < NP / 4; ++i4) {
                        const float4 w = *reinterpret_cast<const float4*>(s_w + o * NP + 4 * i4);
                        dp[4 * i4] += d[e] * w.x; dp[4 * i4 + 1] += d[e] * w.y;
                        dp[4 * i4 + 2] += d[e] * w.z; dp[4 * i4 + 3] += d[e] * w.w;
                    }
                }
            }
            *reinterpret_cast<float4*>(s_u + tid * S::LDU + o4) = make_float4(d[0], d[1], d[2], d[3]);
            *reinterpret_cast<float4*>(s_a + tid * S::LDU + o4) = make_float4(tail_act<ARCH>(a2[o4]), tail_act<ARCH>(a2[o4 + 1]),
                                                                              tail_act<ARCH>(a2[o4 + 2]), tail_act<ARCH>(a2[o4 + 3]));
        }
#pragma unroll
        for (int i4 = 0; i4 < NP; i4 += 4)
            *reinterpret_cast<float4*>(s_v + tid * S::LDV + i4) = make_float4(tail_act<ARCH>(in[i4]), tail_act<ARCH>(in[i4 + 1]),
                                                                              tail_act<ARCH>(in[i4 + 2]), tail_act<ARCH>(in[i4 + 3]));
        s_y[tid] = dy;
#pragma unroll
        for (int q = 0; q < L1 / 4; ++q) {
            const float4 x = pos >= 0 ? row[q] : make_float4(0.f, 0.f, 0.f, 0.f);  // the signs of the squared inputs
            const float xv[4] = {x.x, x.y, x.z, x.w};
            float dv[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int i = 4 * q + e;
                if (ARCH != 0) dv[e] = tail_act_grad<ARCH>(in[i], dp[i]);
                else if (i < L1E) {
                    const float ds = tail_act_grad<0>(in[i], dp[i]), dm = tail_act_grad<0>(in[L1E + i], dp[L1E + i]);
                    // which of the two products is rounded first: as in L3, l1 = 32 has its own form
                    const float k = __fmul_rn(__fmul_rn(2.0f, xv[e]), L1_SQR_SCALE);
                    dv[e] = L1 <= 16 ? __fadd_rn(dm, __fmul_rn(k, ds)) : __fmaf_rn(k, ds, dm);
                } else dv[e] = dy;
            }
            const float4 v = make_float4(dv[0], dv[1], dv[2], dv[3]);
            if (pos >= 0) reinterpret_cast<float4*>(dl1_rows + (size_t)pos * L1)[q] = v;
            *reinterpret_cast<float4*>(s_d + tid * S::LDD + 4 * q) = v;
        }
        __syncthreads();

        if (i0 < NP) {
#pragma unroll 4
            for (int r = 0; r < n; ++r) {
                const float4 du = *reinterpret_cast<const float4*>(s_u + r * S::LDU + o0);
                float v[IT];
#pragma unroll
                for (int b = 0; b < IT; ++b) v[b] = s_v[r * S::LDV + i0 + b];
#pragma unroll
                for (int b = 0; b < IT; ++b) {
                    acc[0][b] += du.x * v[b]; acc[1][b] += du.y * v[b];
                    acc[2][b] += du.z * v[b]; acc[3][b] += du.w * v[b];
                }
            }
        }
#pragma unroll
        for (int j = 0; j < NS; ++j) {
            const int c = tid + j * T;
            if (c >= S::NB) break;
            float sum = other[j];
            if (c < L2) for (int r = 0; r < n; ++r) sum += s_u[r * S::LDU + c];
            else if (c < 2 * L2) for (int r = 0; r < n; ++r) sum += s_a[r * S::LDU + c - L2] * s_y[r];
            else if (c == 2 * L2) for (int r = 0; r < n; ++r) sum += s_y[r];
            else for (int r = 0; r < n; ++r) sum += s_d[r * S::LDD + c - 2 * L2 - 1];
            other[j] = sum;
        }
    }
    block_loss_partial(e2, loss_partials);
    if (!backward) return;
    if (i0 < NP) {
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int b = 0; b < IT; ++b)
                if (i0 + b < NIN) part[ARCH == 0 ? (o0 + a) * NIN + i0 + b : (i0 + b) * L2 + o0 + a] = acc[a][b];
    }
#pragma unroll
    for (int j = 0; j < NS; ++j)
        if (tid + j * T < S::NB) part[S::NW + tid + j * T] = other[j];
}

// Sums of the runs' rows, of a bucket or of the Simple net, in the order of a warp whose lane l adds the rows l, l + 32, .. and
// that then adds across its lanes in halves (l and l + 16, ..).  A thread per cell here, so that the rows are read whole: of the 32
// lanes' sums, eight thread groups take those with l mod 8 = their number, and the first one adds theirs.  blockIdx.y: the
// bucket, or n_seg for the shared L1 bias, the sum over the buckets, of positions with a bucket id out of range too (the last
// segment, which has no gradient of its own).
template <int SPLIT>
__global__ void __launch_bounds__(256) k_tail_wgrad_final(const float* __restrict__ partials, int n_seg, int n_real, int n_cells, int nW,
                                                          int l2, int l1, float* __restrict__ gw2, float* __restrict__ gb2,
                                                          float* __restrict__ gw3, float* __restrict__ gb3, float* __restrict__ gb1,
                                                          float* __restrict__ gb1_shared) {
    __shared__ float s_sum[TB_MAX_BUCKETS + 1][8][32];
    const int g = blockIdx.y, lane = threadIdx.x & 31, group = threadIdx.x >> 5;
    const bool all = g == n_seg;
    const int cell = (all ? nW + 2 * l2 + 1 : 0) + blockIdx.x * 32 + lane;
    const int g0 = all ? 0 : g, g1 = all ? n_seg : g + 1;
    if (cell < n_cells) {
#pragma unroll 5
        for (int q = g0; q < g1; ++q) {
            const float* p = partials + ((size_t)q * SPLIT + group) * n_cells + cell;
            float t[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {  // lane group + 8 j
                t[j] = 0.f;
#pragma unroll
                for (int r = 8 * j; r < SPLIT; r += 32) t[j] += p[(size_t)r * n_cells];
            }
            s_sum[q - g0][group][lane] = (t[0] + t[2]) + (t[1] + t[3]);
        }
    }
    __syncthreads();
    if (group != 0 || cell >= n_cells) return;
    float sum = 0.f;
    for (int q = g0; q < g1; ++q) {
        float t[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) t[j] = s_sum[q - g0][j][lane];
        const float one = ((t[0] + t[4]) + (t[2] + t[6])) + ((t[1] + t[5]) + (t[3] + t[7]));
        sum = all ? sum + one : one;
    }
    if (all) gb1_shared[cell - (nW + 2 * l2 + 1)] = sum;
    else if (g >= n_real) return;
    else if (cell < nW) gw2[(size_t)g * nW + cell] = sum;
    else if (cell < nW + l2) gb2[g * l2 + (cell - nW)] = sum;
    else if (cell < nW + 2 * l2) gw3[g * l2 + (cell - nW - l2)] = sum;
    else if (cell == nW + 2 * l2) gb3[g] = sum;
    else gb1[g * l1 + (cell - nW - 2 * l2 - 1)] = sum;
}

bool tail_tiled(int l1, int l2) { return (l1 == 8 || l1 == 16 || l1 == 32) && (l2 == 16 || l2 == 32); }
// Without the weight gradients the runs are no more than blocks of a launch: a batch of a few positions gets fewer.
static int tail_runs(int arch, int n_pos, int backward) {
    const int runs = arch == 0 ? TB_RUNS_LS : TB_RUNS_SIMPLE;
    return backward || n_pos >= 64 * runs ? runs : n_pos < 64 ? 1 : n_pos / 64;
}
int tail_blocks(int arch, int nb, int n_pos, int backward) { return (arch == 0 ? nb + 1 : 1) * tail_runs(arch, n_pos, backward); }

int launch_tail(cudaStream_t s, int arch, int n_pos, const float* l1_rows, const int* order, const int* seg_start, const float* score,
                const float* wdl, const float* l2_w, const float* l2_b, const float* l3_w, const float* l3_b, LossParams lp, int l1, int l2,
                int nb, float* net_output, float* dy, float* dl1, float* partials, double* loss_partials, int backward) {
    const int blocks = tail_blocks(arch, nb, n_pos, backward), split = tail_runs(arch, n_pos, backward);
#define TAIL_LAUNCH(A, L1, L2, T)                                                                                                 \
    do {                                                                                                                          \
        typedef TailShape<A, L1, L2, T> S;                                                                                        \
        const size_t smem = sizeof(float) * (S::W_FLOATS + (backward ? S::STAGE : 0));                                            \
        cudaFuncSetAttribute(k_tail<A, L1, L2, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(sizeof(float) * (S::W_FLOATS + S::STAGE))); \
        k_tail<A, L1, L2, T><<<blocks, T, smem, s>>>(l1_rows, order, seg_start, split, score, wdl, l2_w, l2_b, l3_w, l3_b, lp, nb, \
                                                     net_output, dy, dl1, partials, loss_partials, backward);                     \
    } while (0)
    // Threads for the positions of an average run.  A warp for up to 32 (16 384 positions of a LayerStack net: 19.4 us, 21.5 with
    // two, 24 with four); for a few positions two, since what is left is the bucket's weights coming in (1024 positions: 25.4 to
    // 23.0).  Up to 56 two: with four a LayerStack net's blocks take a second wave (23 312 positions: 30.6 to 22.8).  A Simple net's full batch, runs of 512, in rounds of 256: 46 us against 52 with 128.
    const int run = n_pos / blocks;
#define TAIL_T(A, L1, L2)                                                                                                         \
    do {                                                                                                                          \
        if (run > 8 && run <= 32 && !(A == 0 && L1 == 32)) TAIL_LAUNCH(A, L1, L2, (A == 0 && L1 == 32 ? 64 : 32));                \
        else if (run <= 56) TAIL_LAUNCH(A, L1, L2, 64);                                                                           \
        else if (A == 0 || run <= 128) TAIL_LAUNCH(A, L1, L2, 128);                                                               \
        else TAIL_LAUNCH(A, L1, L2, (A == 0 ? 128 : 256));                                                                        \
    } while (0)
#define TAIL_L2(A, L1) do { if (l2 == 32) TAIL_T(A, L1, 32); else TAIL_T(A, L1, 16); } while (0)
#define TAIL_L1(A) do { if (l1 == 8) TAIL_L2(A, 8); else if (l1 == 16) TAIL_L2(A, 16); else TAIL_L2(A, 32); } while (0)
    if (arch == 0) TAIL_L1(0); else if (arch == 1) TAIL_L1(1); else TAIL_L1(2);
#undef TAIL_L1
#undef TAIL_L2
#undef TAIL_T
#undef TAIL_LAUNCH
    return 1;
}

int launch_tail_wgrad(cudaStream_t s, int arch, const float* partials, int l1, int l2, int nb, float* gw2, float* gb2, float* gw3, float* gb3,
                      float* gb1, float* gb1_shared) {
    const int nin = arch == 0 ? 2 * (l1 - 1) : l1, nW = nin * l2, n_cells = nW + 2 * l2 + 1 + l1;
    const int n_seg = arch == 0 ? nb + 1 : 1, n_real = arch == 0 ? nb : 1;
    const dim3 grid(ceil_div(n_cells, 32), n_seg + (gb1_shared ? 1 : 0));
    if (arch == 0) k_tail_wgrad_final<TB_RUNS_LS><<<grid, 256, 0, s>>>(partials, n_seg, n_real, n_cells, nW, l2, l1, gw2, gb2, gw3, gb3, gb1, gb1_shared);
    else k_tail_wgrad_final<TB_RUNS_SIMPLE><<<grid, 256, 0, s>>>(partials, n_seg, n_real, n_cells, nW, l2, l1, gw2, gb2, gw3, gb3, gb1, gb1_shared);
    return 1;
}
