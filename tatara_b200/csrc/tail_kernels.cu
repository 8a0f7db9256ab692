// The hidden layers behind L1 in one kernel: L1 activation .. L2 .. L3 .. loss, back to the L1 output, and the block's share of
// the weight gradients of L2, L3 and the biases (trainer_layerstack.rs:2530-2717 forward, :2976-3325 backward;
// trainer_simple.rs:1281-1508, :1560-1765; weight gradients dense_mm_bucket.rs:112-161).  For l1 = 8, 16, 32 and l2 = 16, 32;
// dense_kernels.cu has the kernels for other sizes.
//
// A block owns up to 128 consecutive positions of the bucket order (one bucket), a thread one of them.  The bucket's weights sit in
// shared memory and reach the threads as broadcasts, the position's vectors stay in registers; for the weight gradients the
// threads put them side by side in shared memory and then own cells of the gradient instead.  What bounds it is the latency
// of one block (a single wave covers 65 536 positions); the only large traffic is the L1 rows in and out.  A warp per position
// with every bucket's weights in each block, and the weight gradients in a kernel of their own that read the vectors back
// from memory, took 69 + 74 us at 65 536 positions (LayerStack, l1 = 16), 65 + 92 us (Simple), 23 + 29 us at 1024.
#include "common.cuh"
#include "loss.cuh"

#define TT_POS 128
static_assert(2 * TT_POS == TB_UNIT_TILES * TB_TILE_M, "a block owns half a work unit at most");

namespace {

// ARCH: 0 LayerStack, 1 Simple CReLU (and Pairwise), 2 Simple SCReLU
template <int ARCH, int L1, int L2>
struct TailShape {
    static constexpr int L1E = L1 - 1;
    static constexpr int NIN = ARCH == 0 ? 2 * L1E : L1;  // inputs of L2
    static constexpr int NP = (NIN + 3) / 4 * 4;          // padded
    static constexpr int LDV = NP + 4, LDU = L2 + 4, LDD = L1 + 4;  // row strides: a quarter warp's 16-byte rows hit all banks
    static constexpr int W_FLOATS = L2 * NP + 2 * L2;
    static constexpr int STAGE = TT_POS * (LDV + 2 * LDU + LDD + 1);
    static constexpr int NW = NIN * L2;
    static constexpr int CELLS = NW + 2 * L2 + 1 + L1;
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

template <int ARCH, int L1, int L2>
__global__ void __launch_bounds__(TT_POS) k_tail(const float* __restrict__ l1_rows, const int* __restrict__ order,
                                                 const TileDesc* __restrict__ tiles, const TileDesc* __restrict__ units,
                                                 const int* __restrict__ n_units, int half_tiles, const float* __restrict__ score,
                                                 const float* __restrict__ wdl, const float* __restrict__ l2_w,
                                                 const float* __restrict__ l2_b, const float* __restrict__ l3_w,
                                                 const float* __restrict__ l3_b, LossParams lp, int nb,
                                                 float* __restrict__ net_output, float* __restrict__ dy_out,
                                                 float* __restrict__ dl1_rows, float* __restrict__ partials,
                                                 double* __restrict__ loss_partials, int backward) {
    typedef TailShape<ARCH, L1, L2> S;
    constexpr int NIN = S::NIN, NP = S::NP, L1E = S::L1E;
    extern __shared__ __align__(16) float s_dyn[];
    float* s_w = s_dyn;                    // [L2][NP]
    float* s_b2 = s_w + L2 * NP;           // [L2]
    float* s_w3 = s_b2 + L2;               // [L2]
    float* s_v = s_dyn + S::W_FLOATS;      // [TT_POS][LDV] inputs of L2
    float* s_u = s_v + TT_POS * S::LDV;    // [TT_POS][LDU] gradient of L2's outputs
    float* s_a = s_u + TT_POS * S::LDU;    // [TT_POS][LDU] L2's activations
    float* s_d = s_a + TT_POS * S::LDU;    // [TT_POS][LDD] gradient of the L1 outputs
    float* s_y = s_d + TT_POS * S::LDD;    // [TT_POS] gradient of the output
    const int tid = threadIdx.x;
    const int u = blockIdx.x >> 1, h = blockIdx.x & 1;
    int first = 0, last = 0, g = 0;
    if (u < *n_units) {
        const TileDesc ud = units[u];
        first = ud.start + h * half_tiles;
        last = min(ud.start + ud.count, first + half_tiles);
        g = ud.bucket;
    }
    if (first >= last) {  // nothing here: the sums over the blocks read every row of the units there are
        if (tid == 0) loss_partials[blockIdx.x] = 0.0;
        if (backward && u < *n_units)
            for (int c = tid; c < S::CELLS; c += TT_POS) partials[(size_t)blockIdx.x * S::CELLS + c] = 0.f;
        return;
    }
    const int p_begin = tiles[first].start;
    const int n = tiles[last - 1].start + tiles[last - 1].count - p_begin;
    const bool live = ARCH != 0 || g < nb;  // positions with a bucket id out of range have no L2 and L3
    if (live) {
        const float* w2 = l2_w + (ARCH == 0 ? (size_t)g * S::NW : 0);
        for (int e = tid; e < L2 * NP; e += TT_POS) {
            const int o = e / NP, i = e % NP;
            s_w[e] = i < NIN ? (ARCH == 0 ? w2[o * NIN + i] : w2[i * L2 + o]) : 0.f;
        }
        if (tid < L2) {
            s_b2[tid] = l2_b[(ARCH == 0 ? g * L2 : 0) + tid];
            s_w3[tid] = l3_w[(ARCH == 0 ? g * L2 : 0) + tid];
        }
    }
    const int pos = tid < n ? order[p_begin + tid] : -1;
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
    const float b3 = live ? l3_b[ARCH == 0 ? g : 0] : 0.f;
    __syncthreads();
    float a2[L2];  // L2's clipped outputs
    float out = skip;
    if (live) {
        float l3 = b3;
#pragma unroll
        for (int o = 0; o < L2; ++o) {
            float sum = s_b2[o];
#pragma unroll
            for (int i4 = 0; i4 < NP / 4; ++i4) {
                const float4 w = *reinterpret_cast<const float4*>(s_w + o * NP + 4 * i4);
                const float* x = in + 4 * i4;
                sum += tail_act<ARCH>(x[0]) * w.x; sum += tail_act<ARCH>(x[1]) * w.y;
                sum += tail_act<ARCH>(x[2]) * w.z; sum += tail_act<ARCH>(x[3]) * w.w;
            }
            a2[o] = crelu01(sum);
            l3 += tail_act<ARCH>(a2[o]) * s_w3[o];
        }
        out = ARCH == 0 ? l3 + skip : l3;
    } else {
#pragma unroll
        for (int o = 0; o < L2; ++o) a2[o] = 0.f;
    }
    double e2 = 0.0;
    float dy = 0.f;
    if (pos >= 0) {
        e2 = loss_point(lp, out, sc, wd, &dy);
        net_output[pos] = out;
        dy_out[pos] = dy;
    }
    block_loss_partial(e2, loss_partials);
    if (!backward) return;

    // back to the L1 output; the position's vectors go into shared memory on the way (zeros past the block's positions)
    float dp[NP];
#pragma unroll
    for (int i = 0; i < NP; ++i) dp[i] = 0.f;
#pragma unroll
    for (int o4 = 0; o4 < L2; o4 += 4) {
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
                dv[e] = dm + 2.0f * xv[e] * L1_SQR_SCALE * ds;
            } else dv[e] = dy;
        }
        const float4 v = make_float4(dv[0], dv[1], dv[2], dv[3]);
        if (pos >= 0) reinterpret_cast<float4*>(dl1_rows + (size_t)pos * L1)[q] = v;
        *reinterpret_cast<float4*>(s_d + tid * S::LDD + 4 * q) = v;
    }
    __syncthreads();

    // the block's sums over its positions: a thread owns four outputs and IT inputs of the L2 weights
    float* part = partials + (size_t)blockIdx.x * S::CELLS;
    constexpr int OQ = L2 / 4, G = TT_POS / OQ, IT = (NP + G - 1) / G;
    {
        const int o0 = 4 * (tid % OQ), i0 = IT * (tid / OQ);
        if (i0 < NP) {
            float acc[4][IT];
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int b = 0; b < IT; ++b) acc[a][b] = 0.f;
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
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int b = 0; b < IT; ++b)
                    if (i0 + b < NIN) part[ARCH == 0 ? (o0 + a) * NIN + i0 + b : (i0 + b) * L2 + o0 + a] = acc[a][b];
        }
    }
    // biases of L2, weights of L3, bias of L3, biases of L1
    if (tid < 2 * L2 + 1 + L1) {
        float sum = 0.f;
        if (tid < L2) for (int r = 0; r < n; ++r) sum += s_u[r * S::LDU + tid];
        else if (tid < 2 * L2) for (int r = 0; r < n; ++r) sum += s_a[r * S::LDU + tid - L2] * s_y[r];
        else if (tid == 2 * L2) for (int r = 0; r < n; ++r) sum += s_y[r];
        else for (int r = 0; r < n; ++r) sum += s_d[r * S::LDD + tid - 2 * L2 - 1];
        part[S::NW + tid] = sum;
    }
}

// Sums of the blocks' rows per bucket: 32 cells and eight groups of rows a block; group j adds rows j, j + 8, .. of its
// bucket's blocks, then the groups are added in order.  blockIdx.y: the bucket, or n_seg for the shared L1 bias, to which every
// position contributes, also those with a bucket id out of range (the last segment, which has no gradient of its own).
__global__ void __launch_bounds__(256) k_tail_wgrad_final(const float* __restrict__ partials, const int* __restrict__ unit_base, int n_seg,
                                                          int n_real, int n_cells, int nW, int l2, int l1, float* __restrict__ gw2,
                                                          float* __restrict__ gb2, float* __restrict__ gw3, float* __restrict__ gb3,
                                                          float* __restrict__ gb1, float* __restrict__ gb1_shared) {
    __shared__ float s_sum[8][32];
    const int g = blockIdx.y, lane = threadIdx.x & 31, group = threadIdx.x >> 5;
    const bool all = g == n_seg;
    const int cell = (all ? nW + 2 * l2 + 1 : 0) + blockIdx.x * 32 + lane;
    const int r0 = 2 * unit_base[all ? 0 : g], r1 = 2 * unit_base[all ? n_seg : g + 1];
    float sum = 0.f;
    if (cell < n_cells) {
#pragma unroll 8
        for (int r = r0 + group; r < r1; r += 8) sum += partials[(size_t)r * n_cells + cell];
    }
    s_sum[group][lane] = sum;
    __syncthreads();
    if (group != 0 || cell >= n_cells) return;
#pragma unroll
    for (int j = 1; j < 8; ++j) sum += s_sum[j][lane];
    if (all) gb1_shared[cell - (nW + 2 * l2 + 1)] = sum;
    else if (g >= n_real) return;
    else if (cell < nW) gw2[(size_t)g * nW + cell] = sum;
    else if (cell < nW + l2) gb2[g * l2 + (cell - nW)] = sum;
    else if (cell < nW + 2 * l2) gw3[g * l2 + (cell - nW - l2)] = sum;
    else if (cell == nW + 2 * l2) gb3[g] = sum;
    else gb1[g * l1 + (cell - nW - 2 * l2 - 1)] = sum;
}

bool tail_tiled(int l1, int l2) { return (l1 == 8 || l1 == 16 || l1 == 32) && (l2 == 16 || l2 == 32); }
size_t tail_partial_floats(int arch, int l1, int l2, int max_tiles) {
    const int nin = arch == 0 ? 2 * (l1 - 1) : l1;
    return (size_t)2 * sort_max_units(max_tiles) * (nin * l2 + 2 * l2 + 1 + l1);
}
int tail_loss_blocks(int n_pos) { return 2 * sort_units(n_pos); }

int launch_tail(cudaStream_t s, int arch, int n_pos, const float* l1_rows, const int* order, const TileDesc* tiles, const int* n_tiles, int max_tiles,
                const float* score, const float* wdl, const float* l2_w, const float* l2_b, const float* l3_w, const float* l3_b,
                LossParams lp, int l1, int l2, int nb, float* net_output, float* dy, float* dl1, float* partials,
                double* loss_partials, int backward) {
    const int blocks = tail_loss_blocks(n_pos);
    const TileDesc* units = tiles + max_tiles;
#define TAIL_LAUNCH(A, L1, L2)                                                                                                    \
    do {                                                                                                                          \
        typedef TailShape<A, L1, L2> S;                                                                                           \
        const size_t smem = sizeof(float) * (S::W_FLOATS + (backward ? S::STAGE : 0));                                            \
        cudaFuncSetAttribute(k_tail<A, L1, L2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(sizeof(float) * (S::W_FLOATS + S::STAGE))); \
        k_tail<A, L1, L2><<<blocks, TT_POS, smem, s>>>(l1_rows, order, tiles, units, n_tiles + 1, unit_tiles(n_pos) / 2, score, wdl, l2_w, l2_b, l3_w,   \
                                                       l3_b, lp, nb, net_output, dy, dl1, partials, loss_partials, backward);     \
    } while (0)
#define TAIL_L2(A, L1) do { if (l2 == 32) TAIL_LAUNCH(A, L1, 32); else TAIL_LAUNCH(A, L1, 16); } while (0)
#define TAIL_L1(A) do { if (l1 == 8) TAIL_L2(A, 8); else if (l1 == 16) TAIL_L2(A, 16); else TAIL_L2(A, 32); } while (0)
    if (arch == 0) TAIL_L1(0); else if (arch == 1) TAIL_L1(1); else TAIL_L1(2);
#undef TAIL_L1
#undef TAIL_L2
#undef TAIL_LAUNCH
    return 1;
}

int launch_tail_wgrad(cudaStream_t s, int arch, const float* partials, const int* n_tiles, int l1, int l2, int nb, float* gw2, float* gb2,
                      float* gw3, float* gb3, float* gb1, float* gb1_shared) {
    const int nin = arch == 0 ? 2 * (l1 - 1) : l1, nW = nin * l2, n_cells = nW + 2 * l2 + 1 + l1;
    const int n_seg = nb + 1, n_real = arch == 0 ? nb : 1;
    k_tail_wgrad_final<<<dim3(ceil_div(n_cells, 32), n_seg + (gb1_shared ? 1 : 0)), 256, 0, s>>>(
        partials, n_tiles + 2, n_seg, n_real, n_cells, nW, l2, l1, gw2, gb2, gw3, gb3, gb1, gb1_shared);
    return 1;
}
