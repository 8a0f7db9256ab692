// PackedSfenValue records: device-side decode + feature extraction, host-side encoder and the seeded
// synthetic position generator used by the benchmark and the tests.
//
// Record layout (crates/shogi-format/src/packed_sfen.rs:251-271): bytes 0..31 a bit stream read LSB
// first (side to move, two 7-bit king squares, Huffman-coded board, then hand pieces up to bit 256),
// 32..33 score i16 LE, 34..35 move, 36..37 ply u16 LE, 38 result i8, 39 padding.
#include "common.cuh"
#include "../../include/tatara_b200.h"

#include <math.h>
#include <string.h>

#include <mutex>
#include <vector>

#include "host_mem.cuh"

namespace {

// Huffman table, indexed by code id: none, pawn, lance, knight, silver, bishop, rook, gold
// (packed_sfen.rs:26-35); piece types use the reference's numbering (types.rs: pawn 1, lance 2,
// knight 3, silver 4, bishop 5, rook 6, gold 7, king 8, promoted = +8 for pawn..silver, horse 13, dragon 14).
const unsigned char h_huff_pattern[8] = {0x00, 0x01, 0x03, 0x0b, 0x07, 0x1f, 0x3f, 0x0f};
const unsigned char h_huff_bits[8] = {1, 2, 4, 4, 4, 6, 6, 5};
// board-piece base of the feature index by piece type: {enemy, friend} (bona_piece.rs:59-90)
__constant__ unsigned short d_piece_base[15][2] = {{0, 0},     {171, 90},   {333, 252},   {495, 414},   {657, 576},
                                                   {981, 900}, {1305, 1224}, {819, 738},   {0, 0},       {819, 738},
                                                   {819, 738}, {819, 738},   {819, 738},   {1143, 1062}, {1467, 1386}};
// hand-piece base by hand slot (pawn, lance, knight, silver, gold, bishop, rook): {enemy, friend}
__constant__ unsigned short d_hand_base[7][2] = {{20, 1}, {44, 39}, {54, 49}, {64, 59}, {74, 69}, {82, 79}, {88, 85}};
// emission order of board pieces (types.rs:271-285)
__constant__ unsigned char d_board_piece_types[13] = {1, 2, 3, 4, 7, 5, 6, 9, 10, 11, 12, 13, 14};

struct FsSpec {
    int kings;   // 0 none, 1 two planes, 2 merged plane
    int mirror;  // king-file mirroring (45 king buckets)
    int piece_inputs;
    int max_active;
};

inline bool fs_spec(int feature_set, FsSpec* s) {
    switch (feature_set) {
        case 0: *s = {0, 0, 1548, 38}; return true;
        case 1: *s = {1, 0, 1710, 40}; return true;
        case 2: *s = {2, 0, 1629, 40}; return true;
        case 3: *s = {1, 1, 1710, 40}; return true;
        case 4: *s = {2, 1, 1629, 40}; return true;
    }
    return false;
}

// Next piece code of the Huffman stream (packed_sfen.rs:26-35), from the bits at the stream's position on: the codes are
// told apart by the number t of leading one bits (none 0; pawn 10; lance 1100, knight 1101; silver 1110; gold 11110; bishop
// 111110, rook 111111, first bit lowest), and only t = 2 needs one bit more.  Code ids are piece types: pawn, lance, knight,
// silver, bishop, rook, gold.
__device__ __forceinline__ int huff_decode(unsigned bits, int* len) {
    const int t = __ffs(~bits | 64u) - 1;
    *len = (0x6654421u >> (4 * t)) & 15;
    return ((0x6574210u >> (4 * t)) & 15) + (t == 2 ? (int)((bits >> 3) & 1u) : 0);
}

struct Persp {
    int king_bucket;
    int mirror;
    int color;
};

__device__ __forceinline__ Persp make_persp(const FsSpec& s, int king_sq, int color) {
    const int k = color == 0 ? king_sq : 80 - king_sq;
    Persp p;
    p.color = color;
    if (!s.mirror) {
        p.king_bucket = k;
        p.mirror = 0;
    } else {
        const int file = k / 9, rank = k % 9;
        p.king_bucket = (file >= 5 ? 8 - file : file) * 9 + rank;
        p.mirror = file >= 5;
    }
    return p;
}

// feature index of one packed piece value (feature_set.rs:842-845, :972-991)
__device__ __forceinline__ int feat_index(const FsSpec& s, const Persp& p, int bp) {
    if (p.mirror && bp >= 90) {
        const int rel = bp - 90;
        const int piece = rel / 81, sq = rel % 81;
        bp = 90 + piece * 81 + (8 - sq / 9) * 9 + sq % 9;
    }
    if (s.kings == 2 && bp >= 1629) bp -= 81;
    return p.king_bucket * s.piece_inputs + bp;
}

// What a feature slot holds, before it is turned into the index of either perspective (16 bits): a board piece
// (piece type * 2 + colour) << 7 | square, the perspective's own king or the other one, the i-th piece of a hand
#define SLOT_KING 0x8000u
#define SLOT_HAND 0x4000u
#define SLOT_NONE 0xFFFFu

// Emission order: board pieces by (piece type, colour, ascending square), the friend and enemy king (when the feature set
// has king planes), hand pieces of Black then White by type and count (feature_set.rs:655-808).  Slots >= nnz are filled
// with -1.
//
// A block does PSV_RECORDS records.  One warp decodes, a lane per record: a serial walk of the bit stream, so what bounds
// the kernel is the latency of one record; the stream lives in two registers that are refilled a word at a time and every
// per-record table in shared memory (in local memory, with a table search per symbol, the walk took 100 us).  Then all
// warps expand the slots to both perspectives' indices, a warp per record, so that the index rows leave in 128-byte
// pieces.
#define PSV_RECORDS 32
#define PSV_THREADS 128
__global__ void __launch_bounds__(PSV_THREADS) k_psv_extract(const unsigned* __restrict__ psv, long long n, FsSpec spec,
                                                      int* __restrict__ stm_out, int* __restrict__ nstm_out,
                                                      int* __restrict__ nnz_out, int* __restrict__ bucket_out,
                                                      float* __restrict__ score_out, float* __restrict__ wdl_out) {
    __shared__ unsigned s_raw[PSV_RECORDS * 10];
    __shared__ unsigned short s_piece[81][PSV_RECORDS];  // board pieces in square order
    __shared__ unsigned char s_cnt[30][PSV_RECORDS];     // per (piece type, colour): pieces, then the group's next slot
    __shared__ unsigned short s_slot[PSV_RECORDS][64];
    __shared__ int s_stm[PSV_RECORDS], s_king[PSV_RECORDS][2];
    const long long rec0 = blockIdx.x * (long long)PSV_RECORDS;
    const int n_here = (int)min((long long)PSV_RECORDS, n - rec0);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int A = spec.max_active;
    for (int i = threadIdx.x; i < n_here * 10; i += PSV_THREADS) s_raw[i] = psv[rec0 * 10 + i];
    for (int i = threadIdx.x; i < PSV_RECORDS * 64; i += PSV_THREADS) (&s_slot[0][0])[i] = SLOT_NONE;
    for (int i = threadIdx.x; i < PSV_RECORDS * 30; i += PSV_THREADS) (&s_cnt[0][0])[i] = 0;
    __syncthreads();
    if (warp == 0 && lane < n_here) {
        const unsigned* w = s_raw + lane * 10;
        // the next `have` bits of the stream; past its 256 bits it reads zeros
        unsigned long long buf = w[0] | ((unsigned long long)w[1] << 32);
        int have = 64, next = 2, cur = 0;
        auto take = [&](int k) { buf >>= k; have -= k; cur += k; };
        auto refill = [&]() {
            if (have <= 32) {
                if (next < 8) buf |= (unsigned long long)w[next] << have;
                ++next;
                have += 32;
            }
        };
        const int stm = (int)(buf & 1u), bk = (int)((buf >> 1) & 127u), wk = (int)((buf >> 8) & 127u);
        take(15);
        int n_board = 0;
        for (int sq = 0; sq < 81; ++sq) {
            if (sq == bk || sq == wk) continue;
            refill();
            int len;
            const int id = huff_decode((unsigned)buf, &len);
            if (id == 0) { take(1); continue; }
            // behind the code: the promotion bit (not for gold), then the colour
            const unsigned tail = (unsigned)(buf >> len);
            const int promoted = id != 7 ? (int)(tail & 1u) : 0;
            const int color = (int)((id != 7 ? tail >> 1 : tail) & 1u);
            take(len + (id != 7 ? 2 : 1));
            const int pt = promoted ? (id <= 4 ? id + 8 : (id == 5 ? 13 : 14)) : id;
            const int g = pt * 2 + color;
            s_piece[n_board++][lane] = (unsigned short)(g << 7 | sq);
            s_cnt[g][lane]++;
        }
        unsigned long long hand[2] = {0ull, 0ull};  // a byte per hand slot
        while (cur < 256) {
            refill();
            int len;
            const int id = huff_decode((unsigned)buf << 1 | 1u, &len);  // hand codes leave out the first bit
            const unsigned tail = (unsigned)(buf >> (len - 1));
            const int piecebox = id != 7 ? (int)(tail & 1u) : 0;
            const int color = (int)((id != 7 ? tail >> 1 : tail) & 1u);
            take(len - 1 + (id != 7 ? 2 : 1));
            if (piecebox) continue;  // piece-box entries (handicap games) are not hand pieces
            // hand order pawn, lance, knight, silver, gold, bishop, rook (types.rs Hand::piece_index)
            const unsigned long long one = 1ull << (8 * ((0x46532100u >> (4 * id)) & 15));
            if (color) hand[1] += one; else hand[0] += one;
        }
        int count = 0;
        const int stm_king = stm == 0 ? bk : wk, nstm_king = stm == 0 ? wk : bk;
        if (stm_king < 81 && nstm_king < 81) {
            int run = 0;
            for (int t = 0; t < 13; ++t)
                for (int c = 0; c < 2; ++c) {
                    const int g = d_board_piece_types[t] * 2 + c;
                    const int k = s_cnt[g][lane];
                    s_cnt[g][lane] = (unsigned char)run;
                    run += k;
                }
            for (int i = 0; i < n_board; ++i) {
                const unsigned short piece = s_piece[i][lane];
                const int slot = s_cnt[piece >> 7][lane]++;
                if (slot < A) s_slot[lane][slot] = piece;
            }
            count = min(run, A);
            if (spec.kings != 0) {
                if (count < A) s_slot[lane][count++] = SLOT_KING;
                if (count < A) s_slot[lane][count++] = SLOT_KING | 1;
            }
            for (int owner = 0; owner < 2; ++owner)
                for (int slot = 0; slot < 7; ++slot) {
                    const int nh = (int)(hand[owner] >> (8 * slot)) & 255;
                    for (int i = 0; i < nh && count < A; ++i) s_slot[lane][count++] = (unsigned short)(SLOT_HAND | slot << 8 | owner << 7 | i);
                }
        }
        s_stm[lane] = stm;
        s_king[lane][0] = bk;
        s_king[lane][1] = wk;
        const long long rec = rec0 + lane;
        nnz_out[rec] = count;
        const short score = (short)(w[8] & 0xffffu);
        const signed char result = (signed char)((w[9] >> 16) & 0xffu);
        score_out[rec] = (float)score;
        wdl_out[rec] = result > 0 ? 1.0f : (result < 0 ? 0.0f : 0.5f);
        if (bucket_out) {
            // kingrank9 (crates/shogi-features/src/kingrank9.rs:11-24)
            const int friendly = stm == 0 ? bk : 80 - wk;
            const int enemy = stm == 0 ? 80 - wk : bk;
            bucket_out[rec] = ((friendly % 9) / 3) * 3 + (enemy % 9) / 3;
        }
    }
    __syncthreads();
    for (int r = warp; r < n_here; r += PSV_THREADS / 32) {
        const int stm = s_stm[r];
        for (int p = 0; p < 2; ++p) {
            const int pc = stm ^ p;  // the perspective's colour
            const int own = s_king[r][pc], other = s_king[r][pc ^ 1];
            const Persp ps = make_persp(spec, own, pc);
            int* out = (p ? nstm_out : stm_out) + (rec0 + r) * A;
            for (int slot = lane; slot < A; slot += 32) {
                const unsigned c = s_slot[r][slot];
                int f = -1;
                if (c != SLOT_NONE) {
                    int bp;
                    if (c & SLOT_KING) {
                        const int sq = c & 1u ? other : own;
                        bp = (c & 1u ? 1629 : 1548) + (pc == 0 ? sq : 80 - sq);
                    } else if (c & SLOT_HAND) {
                        bp = d_hand_base[(c >> 8) & 7u][(int)((c >> 7) & 1u) == pc] + (int)(c & 127u);
                    } else {
                        const int sq = c & 127u;
                        bp = d_piece_base[c >> 8][(int)((c >> 7) & 1u) == pc] + (pc == 0 ? sq : 80 - sq);
                    }
                    f = feat_index(spec, ps, bp);
                }
                out[slot] = f;
            }
        }
    }
}

// host loops and the trainer call this with device pointers
void psv_extract_on(cudaStream_t s, const FsSpec& spec, const unsigned* psv, long long n, int* stm, int* nstm, int* nnz, int* bucket,
                    float* score, float* wdl) {
    k_psv_extract<<<(unsigned)((n + PSV_RECORDS - 1) / PSV_RECORDS), PSV_THREADS, 0, s>>>(psv, n, spec, stm, nstm, nnz, bucket, score, wdl);
}

struct BitWriter {
    uint8_t* data;
    int cur;
    void put(unsigned v, int n) {
        for (int i = 0; i < n; ++i, ++cur)
            if ((v >> i) & 1u) data[cur >> 3] |= (uint8_t)(1u << (cur & 7));
    }
};

int huff_id_of(int base_pt) {
    switch (base_pt) {
        case 1: return 1; case 2: return 2; case 3: return 3; case 4: return 4;
        case 5: return 5; case 6: return 6; case 7: return 7;
    }
    return 0;
}

struct SplitMix64 {
    uint64_t s;
    uint64_t next() {
        uint64_t z = (s += 0x9E3779B97F4A7C15ull);
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        return z ^ (z >> 31);
    }
    double unit() { return (double)(next() >> 11) * (1.0 / 9007199254740992.0); }
    uint32_t below(uint32_t n) { return (uint32_t)(((next() >> 32) * (uint64_t)n) >> 32); }
};

}  // namespace

extern "C" int tb_psv_encode(const uint8_t* board_pt, const uint8_t* board_color, const uint8_t* hand_black7,
                             const uint8_t* hand_white7, int side_to_move, int black_king_sq, int white_king_sq,
                             int score, int ply, int result, uint8_t* out) {
    if (!board_pt || !board_color || !hand_black7 || !hand_white7 || !out) return TB_ERR_INVALID_ARGUMENT;
    memset(out, 0, 40);
    BitWriter bw{out, 0};
    bw.put((unsigned)side_to_move & 1u, 1);
    bw.put((unsigned)black_king_sq, 7);
    bw.put((unsigned)white_king_sq, 7);
    for (int sq = 0; sq < 81; ++sq) {
        if (sq == black_king_sq || sq == white_king_sq) continue;
        int pt = board_pt[sq];
        if (pt == 0) { bw.put(0, 1); continue; }
        int promoted = 0, base = pt;
        if (pt >= 9 && pt <= 12) { promoted = 1; base = pt - 8; }
        else if (pt == 13) { promoted = 1; base = 5; }
        else if (pt == 14) { promoted = 1; base = 6; }
        const int id = huff_id_of(base);
        if (id == 0) return TB_ERR_INVALID_ARGUMENT;
        bw.put(h_huff_pattern[id], h_huff_bits[id]);
        if (id != 7) bw.put((unsigned)promoted, 1);
        bw.put(board_color[sq] & 1u, 1);
        if (bw.cur > 256) return TB_ERR_INVALID_ARGUMENT;
    }
    // hand pieces: code without its first bit, a piece-box flag of 0 (not for gold), colour
    static const int slot_pt[7] = {1, 2, 3, 4, 7, 5, 6};
    for (int color = 0; color < 2; ++color) {
        const uint8_t* h = color == 0 ? hand_black7 : hand_white7;
        for (int slot = 0; slot < 7; ++slot)
            for (int k = 0; k < h[slot]; ++k) {
                const int id = huff_id_of(slot_pt[slot]);
                bw.put((unsigned)h_huff_pattern[id] >> 1, h_huff_bits[id] - 1);
                if (id != 7) bw.put(0, 1);
                bw.put((unsigned)color, 1);
                if (bw.cur > 256) return TB_ERR_INVALID_ARGUMENT;
            }
    }
    const int16_t sc = (int16_t)score;
    out[32] = (uint8_t)(sc & 0xff);
    out[33] = (uint8_t)((sc >> 8) & 0xff);
    out[36] = (uint8_t)(ply & 0xff);
    out[37] = (uint8_t)((ply >> 8) & 0xff);
    out[38] = (uint8_t)(int8_t)result;
    return TB_OK;
}

// Synthetic positions.  Every record holds the full 40-piece set, which always fills the 256 bits
// exactly.  Drawn from one SplitMix64 stream in this order per record: side to move (1 bit), black
// king square (uniform of 81), white king square (uniform of the other 80); then for each of the 38
// other pieces in the order 18 pawns, 4 lances, 4 knights, 4 silvers, 4 golds, 2 bishops, 2 rooks:
// on the board with p = 0.85 (uniform empty square, uniform owner, promoted with p = 0.1 unless gold),
// otherwise in the hand of a uniform side; score = round(400 * N(0,1)) clipped to +-3000 (Box-Muller);
// result = draw with p = 0.05, else win with p = sigmoid(score / 600), else loss; ply uniform in 1..256.
// Legality of the position is not enforced (the extractor does not need it).
extern "C" int tb_psv_synthesize(uint64_t seed, int64_t n_records, uint8_t* out) {
    if (n_records < 0 || (n_records > 0 && !out)) return TB_ERR_INVALID_ARGUMENT;
    SplitMix64 rng{seed};
    static const int piece_list[7][2] = {{1, 18}, {2, 4}, {3, 4}, {4, 4}, {7, 4}, {5, 2}, {6, 2}};
    for (int64_t r = 0; r < n_records; ++r) {
        uint8_t pt[81] = {0}, col[81] = {0}, hand[2][7] = {{0}};
        const int stm = (int)(rng.next() & 1u);
        const int bk = (int)rng.below(81);
        int wk = (int)rng.below(80);
        if (wk >= bk) ++wk;
        pt[bk] = 8; col[bk] = 0;
        pt[wk] = 8; col[wk] = 1;
        int empties = 79;
        for (int t = 0; t < 7; ++t)
            for (int k = 0; k < piece_list[t][1]; ++k) {
                const int type = piece_list[t][0];
                if (rng.unit() < 0.85) {
                    int pick = (int)rng.below((uint32_t)empties), sq = 0;
                    for (;; ++sq)
                        if (pt[sq] == 0 && pick-- == 0) break;
                    const int owner = (int)(rng.next() & 1u);
                    int placed = type;
                    if (type != 7 && rng.unit() < 0.1) placed = type <= 4 ? type + 8 : (type == 5 ? 13 : 14);
                    pt[sq] = (uint8_t)placed;
                    col[sq] = (uint8_t)owner;
                    --empties;
                } else {
                    const int owner = (int)(rng.next() & 1u);
                    static const int slot_of[8] = {-1, 0, 1, 2, 3, 5, 6, 4};
                    hand[owner][slot_of[type]]++;
                }
            }
        double u1 = rng.unit();
        if (u1 < 1e-300) u1 = 1e-300;
        const double u2 = rng.unit();
        const double z = sqrt(-2.0 * log(u1)) * cos(6.283185307179586 * u2);
        long sc = lrint(z * 400.0);
        if (sc > 3000) sc = 3000;
        if (sc < -3000) sc = -3000;
        int result;
        if (rng.unit() < 0.05) result = 0;
        else result = rng.unit() < 1.0 / (1.0 + exp(-(double)sc / 600.0)) ? 1 : -1;
        const int ply = 1 + (int)rng.below(256);
        const int rc = tb_psv_encode(pt, col, hand[0], hand[1], stm, bk, wk, (int)sc, ply, result, out + 40 * r);
        if (rc != TB_OK) return rc;
    }
    return TB_OK;
}

// Device-to-device form for the trainer: records already in device memory -> step inputs in device memory, on `s`.
// Returns the number of kernels launched, or -1 for an unknown feature set.
int launch_psv_extract(cudaStream_t s, int feature_set, const void* d_psv, long long n, int* stm, int* nstm, int* nnz,
                       int* bucket, float* score, float* wdl) {
    FsSpec spec;
    if (!fs_spec(feature_set, &spec)) return -1;
    if (n <= 0) return 0;
    psv_extract_on(s, spec, static_cast<const unsigned*>(d_psv), n, stm, nstm, nnz, bucket, score, wdl);
    return 1;
}

// dimensions of a feature set id: rows of the FT table, slots per perspective, rows per king bucket (feature_set.rs:1031-1038)
bool psv_feature_set_dims(int feature_set, int* ft_in, int* max_active, int* piece_inputs) {
    FsSpec spec;
    if (!fs_spec(feature_set, &spec)) return false;
    *ft_in = (spec.mirror ? 45 : 81) * spec.piece_inputs;
    *max_active = spec.max_active;
    *piece_inputs = spec.piece_inputs;
    return true;
}

// ---- host records -> host arrays -------------------------------------------------------------------------------------
// A loader calls this for every batch, so what a call works with is kept: two streams, device buffers and page-locked
// staging.  Allocating and freeing them per call took 14 of the 14.4 ms of a 65 536-record call.  At most EXTRACT_KEEP
// sets of EXTRACT_KEEP_BYTES are kept per device; a call takes one for itself, so threads do not share any.
namespace {

#define EXTRACT_KEEP 4
#define EXTRACT_KEEP_BYTES ((size_t)96 << 20)
#define EXTRACT_CHUNK 16384         // records per piece of the pipeline: 5 MB of results, 0.1 ms of copying
#define EXTRACT_CHUNK_STAGED 32768  // through the staging buffer: room for the copying threads
#define EXTRACT_EVENTS 64

struct ExtractCtx {
    int device = 0;
    cudaStream_t s[2] = {nullptr, nullptr};
    cudaEvent_t ev[EXTRACT_EVENTS] = {};
    unsigned char* d_buf = nullptr;  // records, then the results chunk by chunk
    unsigned char* h_buf = nullptr;  // the same layout in page-locked memory
    size_t d_bytes = 0, h_bytes = 0;
};

struct ExtractPool {
    std::mutex mu;
    std::vector<ExtractCtx*> idle;
};
ExtractPool& extract_pool() { static ExtractPool* p = new ExtractPool; return *p; }

void extract_free(ExtractCtx* c) {
    cudaFree(c->d_buf);
    if (c->h_buf) pinned_free(c->h_buf);
    for (cudaEvent_t e : c->ev) if (e) cudaEventDestroy(e);
    for (cudaStream_t s : c->s) if (s) cudaStreamDestroy(s);
    delete c;
}

ExtractCtx* extract_take(int device) {
    {
        ExtractPool& P = extract_pool();
        std::lock_guard<std::mutex> lock(P.mu);
        for (size_t i = P.idle.size(); i-- > 0;)
            if (P.idle[i]->device == device) {
                ExtractCtx* c = P.idle[i];
                P.idle.erase(P.idle.begin() + i);
                return c;
            }
    }
    ExtractCtx* c = new ExtractCtx;
    c->device = device;
    bool ok = true;
    for (cudaStream_t& s : c->s) ok = ok && cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) == cudaSuccess;
    for (cudaEvent_t& e : c->ev) ok = ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
    if (ok) return c;
    extract_free(c);
    return nullptr;
}

void extract_give_back(ExtractCtx* c) {
    std::vector<ExtractCtx*> out;
    if (c->d_bytes > EXTRACT_KEEP_BYTES) {
        out.push_back(c);
    } else {
        ExtractPool& P = extract_pool();
        std::lock_guard<std::mutex> lock(P.mu);
        P.idle.push_back(c);
        int same = 0;
        for (size_t i = P.idle.size(); i-- > 0;)
            if (P.idle[i]->device == c->device && ++same > EXTRACT_KEEP) { out.push_back(P.idle[i]); P.idle.erase(P.idle.begin() + i); }
    }
    for (ExtractCtx* o : out) extract_free(o);
}

cudaError_t extract_reserve(ExtractCtx* c, size_t d_bytes, size_t h_bytes) {
    if (d_bytes > c->d_bytes) {
        cudaFree(c->d_buf);
        c->d_buf = nullptr;
        c->d_bytes = 0;
        const cudaError_t e = cudaMalloc((void**)&c->d_buf, d_bytes);
        if (e != cudaSuccess) return e;
        c->d_bytes = d_bytes;
    }
    if (h_bytes > c->h_bytes) {
        if (c->h_buf) pinned_free(c->h_buf);
        c->h_bytes = 0;
        c->h_buf = static_cast<unsigned char*>(pinned_alloc(h_bytes));
        if (!c->h_buf) return cudaErrorMemoryAllocation;
        c->h_bytes = h_bytes;
    }
    return cudaSuccess;
}

bool page_locked(const void* p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) { cudaGetLastError(); return false; }
    return a.type == cudaMemoryTypeHost;
}

}  // namespace

// frees the idle contexts (memory is short)
void psv_extract_trim() {
    std::vector<ExtractCtx*> out;
    {
        ExtractPool& P = extract_pool();
        std::lock_guard<std::mutex> lock(P.mu);
        out.swap(P.idle);
    }
    for (ExtractCtx* c : out) extract_free(c);
}

extern "C" int tb_psv_extract(int device, int feature_set, const uint8_t* psv, int64_t n, int32_t* stm_indices,
                              int32_t* nstm_indices, int32_t* nnz, int32_t* bucket, float* score, float* wdl) {
    FsSpec spec;
    if (!fs_spec(feature_set, &spec) || n < 0) return TB_ERR_INVALID_ARGUMENT;
    if (n == 0) return TB_OK;
    if (!psv || !stm_indices || !nstm_indices || !nnz || !score || !wdl) return TB_ERR_INVALID_ARGUMENT;
    if (cudaSetDevice(device) != cudaSuccess) return TB_ERR_NO_DEVICE;
    ExtractCtx* c = extract_take(device);
    if (!c) return TB_ERR_CUDA;
    const size_t A = (size_t)spec.max_active;
    const size_t row[6] = {A * 4, A * 4, 4, 4, 4, 4};
    unsigned char* dst[6] = {(unsigned char*)stm_indices, (unsigned char*)nstm_indices, (unsigned char*)nnz, (unsigned char*)bucket,
                             (unsigned char*)score, (unsigned char*)wdl};
    // page-locked arrays are copied into directly; a call with a pageable one, and a small call (where one copy of
    // everything beats six), goes through the staging buffer
    const bool small = (size_t)n * (2 * A + 14) * 4 < ((size_t)1 << 20);
    bool staged = small;
    for (int k = 0; k < 6 && !staged; ++k) staged = dst[k] && !page_locked(dst[k]);
    const bool psv_staged = small || !page_locked(psv);
    const size_t most = staged ? EXTRACT_CHUNK_STAGED : EXTRACT_CHUNK;
    const size_t chunk = (size_t)n < most ? (size_t)n : most, n_chunks = ((size_t)n + chunk - 1) / chunk;
    // results: array by array; with staging in blocks of one chunk (a transfer each), else over all records.  Every array
    // starts on a 16-byte boundary.
    const size_t block = staged ? chunk : (size_t)n;
    size_t off[7] = {0};
    for (int k = 0; k < 6; ++k) off[k + 1] = off[k] + (block * row[k] + 15) / 16 * 16;
    const size_t rec_bytes = ((size_t)n * 40 + 255) / 256 * 256;
    const size_t total = rec_bytes + (staged ? n_chunks : 1) * off[6];
    cudaError_t e = extract_reserve(c, total, staged ? total : psv_staged ? rec_bytes : 0);
    if (e == cudaErrorMemoryAllocation) {  // other calls' idle buffers may be what is missing
        cudaGetLastError();
        psv_extract_trim();
        e = extract_reserve(c, total, staged ? total : psv_staged ? rec_bytes : 0);
    }
    auto chk = [&](cudaError_t x) { if (e == cudaSuccess) e = x; };
    // the host side of chunk i once its results are in the staging buffer
    auto deliver = [&](size_t i) {
        const size_t r0 = i * chunk, r = (size_t)n - r0 < chunk ? (size_t)n - r0 : chunk;
        const unsigned char* src = c->h_buf + rec_bytes + i * off[6];
        HostCopy items[6];
        int m = 0;
        for (int k = 0; k < 6; ++k)
            if (dst[k]) items[m++] = {dst[k] + r0 * row[k], src + off[k], r * row[k]};
        host_copy_out(items, m);
    };
    size_t delivered = 0;
    for (size_t i = 0; i < n_chunks && e == cudaSuccess; ++i) {
        cudaStream_t s = c->s[i & 1];  // two streams: one chunk's records travel down while the other's results travel up
        const size_t r0 = i * chunk, r = (size_t)n - r0 < chunk ? (size_t)n - r0 : chunk;
        const unsigned char* src = psv + r0 * 40;
        if (psv_staged) { host_stage(c->h_buf + r0 * 40, src, r * 40); src = c->h_buf + r0 * 40; }
        chk(cudaMemcpyAsync(c->d_buf + r0 * 40, src, r * 40, cudaMemcpyHostToDevice, s));
        unsigned char* d[6];
        for (int k = 0; k < 6; ++k) d[k] = c->d_buf + rec_bytes + off[k] + (staged ? i * off[6] : r0 * row[k]);
        psv_extract_on(s, spec, (const unsigned*)(c->d_buf + r0 * 40), (long long)r, (int*)d[0], (int*)d[1], (int*)d[2],
                       bucket ? (int*)d[3] : nullptr, (float*)d[4], (float*)d[5]);
        chk(cudaGetLastError());
        if (staged) {
            chk(cudaMemcpyAsync(c->h_buf + rec_bytes + i * off[6], d[0], off[6], cudaMemcpyDeviceToHost, s));
            if (n_chunks > 1) {
                if (i >= EXTRACT_EVENTS) {  // the event's previous chunk is delivered before it is recorded again
                    chk(cudaEventSynchronize(c->ev[delivered % EXTRACT_EVENTS]));
                    if (e == cudaSuccess) deliver(delivered++);
                }
                chk(cudaEventRecord(c->ev[i % EXTRACT_EVENTS], s));
            }
        } else {
            for (int k = 0; k < 2; ++k) chk(cudaMemcpyAsync(dst[k] + r0 * row[k], d[k], r * row[k], cudaMemcpyDeviceToHost, s));
            if (n_chunks > 1) chk(cudaEventRecord(c->ev[i & 1], s));
        }
    }
    if (!staged && e == cudaSuccess) {
        // the narrow arrays in one transfer each, behind the last chunks of both streams
        cudaStream_t s = c->s[(n_chunks - 1) & 1];
        if (n_chunks > 1) chk(cudaStreamWaitEvent(s, c->ev[n_chunks & 1], 0));
        for (int k = 2; k < 6; ++k)
            if (dst[k]) chk(cudaMemcpyAsync(dst[k], c->d_buf + rec_bytes + off[k], (size_t)n * row[k], cudaMemcpyDeviceToHost, s));
    }
    if (staged && n_chunks > 1)
        while (delivered < n_chunks && e == cudaSuccess) {
            chk(cudaEventSynchronize(c->ev[delivered % EXTRACT_EVENTS]));
            if (e == cudaSuccess) deliver(delivered++);
        }
    chk(cudaStreamSynchronize(c->s[0]));
    if (n_chunks > 1) chk(cudaStreamSynchronize(c->s[1]));
    if (staged && n_chunks == 1 && e == cudaSuccess) deliver(0);
    if (e != cudaSuccess) {
        cudaStreamSynchronize(c->s[0]);
        cudaStreamSynchronize(c->s[1]);
        extract_free(c);
        return TB_ERR_CUDA;
    }
    extract_give_back(c);
    return TB_OK;
}
