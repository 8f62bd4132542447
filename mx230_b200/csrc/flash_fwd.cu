// Flash-attention forward for sm_100a: O = softmax(scale * Q K^T [+ causal]) V and
// the per-row log-sum-exp L = m + ln(l), never materialising the N x N scores.
//
// Reference semantics: flash_fwd / attn_flash / attn_flash_lse,
// 02-flash-attention/kernels/attention_flash.cu:17-100 (fp32 SIMT, one thread per
// query row).  This kernel keeps those semantics (scale 1/sqrt(64), key j <= query i
// when causal, any N, natural-log L) and maps the two contractions onto the 5th-gen
// tensor cores:
//
//   * a work item is 256 query rows of one head as two 128-row tiles (or, for calls that would fill the SMs unevenly, one
//     tile with its key tiles split between the softmax groups: KEY_SPLIT below; for calls of few items 64 rows:
//     flash_fwd_rows64_kernel); the kernel is persistent:
//     one CTA per SM walks a fixed share of the items (heaviest first, dealt out in snake order so
//     that every CTA gets the same number of key tiles), and every role runs ahead into the next
//     item on its own, so the next item's Q / K loads and first Q K^T run under the current
//     item's last softmax and its epilogue;
//   * warps 0-15 are four softmax warpgroups, two per query tile (tile t = warp / 8), each taking 64 of
//     the 128 key columns of every score tile, one thread per (query row, half): the thread pulls its
//     columns into registers 32 at a time (the second piece lands under the first one's exponentials),
//     which frees S_t for the next Q K^T, takes exp2 and the row sum, and writes bf16 P into its own
//     tensor-memory columns.  Usually without a row max (see the fixed-reference mode below: the
//     halves of a row then meet only once per item, to add their sums); otherwise the halves exchange
//     their part of the row max through shared memory and O_t is rescaled in tensor memory only when
//     the max grows by > 2^8;
//   * warp 16 streams Q (two buffers, alternating by item) and K/V tiles (128 keys) through a
//     4-stage shared-memory ring with plain per-CTA TMA tile loads (128-byte swizzle);
//   * warp 17 issues the tcgen05.mma stream S_t = Q_t K^T into tensor memory (128 fp32 columns
//     per tile), warp 18 the stream O_t += P_t V with P_t read from tensor memory as bf16 (each
//     stream has its own warp, which runs its loop warp-uniformly with one elected lane issuing).
//   The two tiles ping-pong and S, P, O never alias, so the tensor core computes the next
//   scores and the other tile's P V while a tile's softmax runs on the CUDA cores.
//
// Operands are bf16 (rounded once by the cast pre-pass), accumulation is fp32.
#include <cuda_fp16.h>
#include <math_constants.h>

#include <cstring>
#include <type_traits>

#include "common.cuh"

namespace {

constexpr int BM = 128;        // query rows per tile
constexpr int QT = 2;          // query tiles per CTA
constexpr int BN = 128;        // keys per K/V tile
constexpr int HD = 64;
constexpr int KV_STAGES = 4;
constexpr int TILE_BYTES = BN * HD * 2;  // 16 KB
constexpr int HALVES = 2;               // softmax groups per query tile: each takes half of the tile's key columns
constexpr int SOFT_WARPS = QT * HALVES * 4;   // 16
constexpr int FWD_THREADS = (SOFT_WARPS + 3) * 32;   // 608: four softmax warpgroups + {TMA, 2 MMA issuers}
// No 20th, idle warp and no register moves between warps: every warp runs at the 96 registers per thread of the launch.
// (640 threads, 104 for the softmax warps and 64 for the others by setmaxnreg: 48 x 4096 rows causal 170.8 us a call against
// 166.1, no mask 284.6 against 270.0, bf16 operands 396 against 361, 8 x 8192 rows 176.7 against 164.3.)

// build-time knobs of the softmax loop
#ifndef FWD_FAST
#define FWD_FAST 1        // fixed-reference mode (no row max, no subtraction) while the sums stay in range
#endif
#ifndef FWD_POLY
#define FWD_POLY 1        // of every FWD_POLY_DEN column pairs, how many take 2^x from the FMA-pipe polynomial (with four
                          // softmax warps per scheduler the loop is issue-bound: 1 of 4 beats 2 of 4 by 7-10 %, 0 of 4 loses 9 %)
#endif
#ifndef FWD_POLY_DEN
#define FWD_POLY_DEN 4
#endif
// The MMA issuer warps run warp-uniformly (waits included) with one elected lane issuing.
#define ISSUER_WAIT(w) __all_sync(0xFFFFFFFFu, (w))
#define ISSUER_LANE mx::elect_one()

constexpr int Q_BUFS = 2;                // Q of the next item lands while the current one is in use
constexpr int SMEM_Q = 0;
constexpr int SMEM_K = SMEM_Q + Q_BUFS * QT * TILE_BYTES;
constexpr int SMEM_V = SMEM_K + KV_STAGES * TILE_BYTES;
constexpr int SMEM_BAR = SMEM_V + KV_STAGES * TILE_BYTES;
constexpr int XCH_PUBS = 3;                // groups that hand their row sums over (one per query tile; three in the key-split form)
constexpr int SMEM_XCH = SMEM_BAR + 512;   // [2 item parities][XCH_PUBS][3][BM] floats: row sums (and max) handed to the group that does the epilogue
constexpr int SMEM_XMAX = SMEM_XCH + 2 * XCH_PUBS * 3 * BM * 4;   // [QT][2 tile parities][HALVES][BM] floats: row-max parts of the general mode
constexpr int KSKB_SLOTS = 8;              // int8 scores: ring of the key tiles' scales and offsets
constexpr int KSKB_BYTES = 2 * BN * 4;     // ks[BN], kb[BN]
constexpr int SMEM_KSKB = SMEM_XMAX + QT * 2 * HALVES * BM * 4;
constexpr int SMEM_TOTAL = SMEM_KSKB + KSKB_SLOTS * KSKB_BYTES;
constexpr int SMEM_ALLOC = SMEM_TOTAL + 1024;  // slack for 1024-byte alignment

// barrier slots (8 bytes each) inside SMEM_BAR
constexpr int BAR_Q_FULL = 0;                    // [Q_BUFS]
constexpr int BAR_Q_EMPTY = BAR_Q_FULL + Q_BUFS; // [Q_BUFS] softmax warps -> TMA: item done with its Q buffer
constexpr int BAR_K_FULL = BAR_Q_EMPTY + Q_BUFS; // [KV_STAGES]
constexpr int BAR_K_EMPTY = BAR_K_FULL + KV_STAGES;
constexpr int BAR_V_FULL = BAR_K_EMPTY + KV_STAGES;
constexpr int BAR_V_EMPTY = BAR_V_FULL + KV_STAGES;
constexpr int BAR_S_FULL = BAR_V_EMPTY + KV_STAGES;  // [QT] MMA -> softmax: S_t written
constexpr int BAR_S_FREE = BAR_S_FULL + QT;          // [QT] softmax -> MMA: S_t copied to registers
constexpr int BAR_P_FULL = BAR_S_FREE + QT;          // [QT] softmax -> MMA: P_t written
constexpr int BAR_O_DONE = BAR_P_FULL + QT;          // [QT] MMA -> softmax: O_t += P_t V complete
constexpr int BAR_XCH = BAR_O_DONE + QT;             // [QT] row sums are published (key-split form: [0] only, by three groups)
constexpr int BAR_XMAX = BAR_XCH + QT;               // [QT] both halves of tile t have published their part of the row max (general loop, first tile of REF sources)
constexpr int BAR_O1_READ = BAR_XMAX + QT;           // key-split form: O_1 of the item has been read by the epilogue
constexpr int N_BARS = BAR_O1_READ + 1;
static_assert(8 * N_BARS + 16 <= 512, "barrier area");

// tensor-memory columns: nothing aliases, so S_t(j+1) can be produced while P_t(j) is consumed
constexpr int TM_S = 0;     // S_t at TM_S + t*128, fp32
constexpr int TM_P = 256;   // P_t at TM_P + t*64, bf16 pairs
constexpr int TM_O = 384;   // O_t at TM_O + t*64, fp32
constexpr int TM_COLS = 512;

// The running row max is only raised when it would grow by more than 2^RESCALE_LOG2 in the
// exponent; until then probabilities are taken against the stale max (they stay below
// 2^RESCALE_LOG2, harmless in bf16/fp32) and O needs no rescale.
constexpr float RESCALE_LOG2 = 8.0f;

struct FwdParams {
    float *O;             // row r of head h at O + h*o_head_stride + r*o_row_stride (floats)
    __half *O_half;       // [heads][n_q][64]: the same rows in fp16 for the projection that follows, or null.  May be where Q
                          // is staged: an item's Q tile is read by that item alone, before the first row of its O exists
    float *L;             // [heads][n_q] or null
    long long o_head_stride, o_row_stride;
    int n_q;              // query rows per head
    int n_k;              // keys per head
    int q_off;            // causal: query row r sees keys <= r + q_off (0 for self-attention)
    int kv_group;         // query heads per K/V head (K/V head of query head h is h / kv_group)
    int causal;
    int heads;            // query heads (items are (query block, head) pairs, heads fastest)
    int item_rows;        // query rows per work item: QT*BM, or fewer when such items would leave SMs without work
    int n_qblocks;        // blocks of item_rows query rows per head
    int n_items;          // heads * n_qblocks
    int tma_out;          // O leaves through staged TMA stores (strides and base 16-byte aligned) or per-thread stores
    const float *q_norm2; // [heads][MX230_NORM_PARTS] largest squared row norm of the unscaled Q per head and part, or null
    const float *k_norm2; // [heads / kv_group][MX230_NORM_PARTS] the same for K
    int test_drop_tile;   // test hook: K/V tile (counted over the CTA's items) that CTA 0's producer never requests; -1 = off
    // int8 score mode (prefill over an int8 cache with the reference kernel's arithmetic): Q and K hold int8 CODES
    // (exact in bf16), so the MMA returns exact integer dots, and the score is rebuilt per element as
    // row_a[i] * (dot * ks[j] + row_qsum[i] * kb[j]) in log2 units (03-llm-engine/kernels/llm.cu:3774-3782)
    const float *row_a;      // [heads][n_q]   q scale * 1/sqrt(64) * log2(e), or null = mode off
    const float *row_qsum;   // [heads][n_q]   sum of the row's q codes
    const float *col_kskb;   // [heads / kv_group][key tiles][ks[BN], kb[BN]]: scale and offset of every key
    int n_k_tiles;           // key tiles of BN keys
    int *status;
};

__device__ __forceinline__ float fmax3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// The CTA's `round`-th work item.  Items are listed heaviest first (when causal: the latest query block of
// every head, then the one before, ...) and dealt to the CTAs forwards in even rounds, backwards in odd ones.
__device__ __forceinline__ bool fwd_item(const FwdParams &P, int round, int &bh, int &q0) {
    const int G = (int)gridDim.x, c = (int)blockIdx.x;
    const int i = round * G + ((round & 1) ? G - 1 - c : c);
    if (i >= P.n_items) return false;
    const int rank = i / P.heads;
    bh = i - rank * P.heads;
    q0 = (P.causal ? P.n_qblocks - 1 - rank : rank) * P.item_rows;
    return true;
}
// K/V tiles that query tile `t` of the block starting at row q0 has to see
__device__ __forceinline__ int fwd_tile_iters(const FwdParams &P, int q0, int t) {
    const int r0 = q0 + t * BM;
    if (r0 >= P.n_q || t * BM >= P.item_rows) return 0;
    const int n_kv_total = (P.n_k + BN - 1) / BN;
    return P.causal ? min(n_kv_total, (r0 + BM - 1 + P.q_off) / BN + 1) : n_kv_total;
}

// In front of the wait for the previous kernel: the tensor maps on their way into the SM's caches.
__device__ __forceinline__ void fwd_prefetch_maps(const FwdParams &P, int warp, int lane, const CUtensorMap &tmQ, const CUtensorMap &tmK,
                                                  const CUtensorMap &tmV, const CUtensorMap &tmO) {
    if (warp == SOFT_WARPS && lane == 0) {
        mx::tma_prefetch_desc(&tmQ);
        mx::tma_prefetch_desc(&tmK);
        mx::tma_prefetch_desc(&tmV);
        if (P.tma_out) mx::tma_prefetch_desc(&tmO);
    }
}

// Largest score, in log2 units, of a head that takes the max-free loop: against the reference 0, or (SRC_RAW_BOUND, SRC_I8) against
// a row's max over the first key tile, from which a score may be twice as far (probabilities stay below 2^80 either way).
constexpr float FAST_BOUND = 80.0f, FAST_BOUND_REF = 40.0f;
// Whether every score of head `bh` is within `bound` (see the softmax loop); whole-warp call.  Operands the
// caller staged: from the bound that raw_bounds_kernel left in L at every 64th row (`row0`: the first one of the query tile),
// read before that tile's epilogue, which overwrites it and which waits for every warp that reads it.
__device__ __forceinline__ bool fwd_fast_raw(const FwdParams &P, int bh, int row0) {
    return FWD_FAST && row0 < P.n_q && *(const volatile float *)(P.L + (size_t)bh * P.n_q + row0) <= FAST_BOUND_REF * FAST_BOUND_REF;
}
__device__ __forceinline__ bool fwd_fast_head(const FwdParams &P, int bh, int lane, float bound) {
    if (!FWD_FAST || P.q_norm2 == nullptr) return false;
    static_assert(MX230_NORM_PARTS == 32, "one part per lane");
    // norms are >= 0 or NaN: as integers they order like that, with NaN the largest
    const int nq = __reduce_max_sync(0xFFFFFFFFu, __float_as_int(P.q_norm2[(size_t)bh * MX230_NORM_PARTS + lane]) & 0x7FFFFFFF);
    const int nk = __reduce_max_sync(0xFFFFFFFFu, __float_as_int(P.k_norm2[(size_t)(bh / P.kv_group) * MX230_NORM_PARTS + lane]) & 0x7FFFFFFF);
    // the norms are those of the fp32 values; rounding to bf16 moves a norm by less than 0.4 %
    return __int_as_float(nq) * __int_as_float(nk) * (MX230_QK_LOG2_SCALE * MX230_QK_LOG2_SCALE) <= bound * bound;
}

// Where scores come from: Q staged times scale * log2(e) (they arrive in log2 units), Q and K as the caller gave them
// (general loop only), the same with a bound in L, or int8 codes of both (exact integer dots, see FwdParams::row_a).
// (A kernel of its own for RAW without a bound: with the max-free loop beside it the general one is 5 % slower.)
enum { SRC_PRE = 0, SRC_RAW = 1, SRC_RAW_BOUND = 2, SRC_I8 = 3 };

// int8 scores: exact integer dots -> row_a * (dot * ks + qsum * kb) + add, two keys per instruction
__device__ __forceinline__ void fwd_rebuild32(uint32_t *x, const float *kskb, float add, float row_a, float row_qsum) {
    const uint64_t add_2 = mx::pk2(add, add);
    const uint64_t qs2 = mx::pk2(row_qsum, row_qsum), ra2 = mx::pk2(row_a, row_a);
#pragma unroll
    for (int i = 0; i < 32; i += 4) {
        const float4 k4 = *(const float4 *)(kskb + i), b4 = *(const float4 *)(kskb + BN + i);
        const uint64_t u = mx::fma2(mx::pk2(__uint_as_float(x[i]), __uint_as_float(x[i + 1])), mx::pk2(k4.x, k4.y),
                                    mx::mul2(qs2, mx::pk2(b4.x, b4.y)));
        const uint64_t w = mx::fma2(mx::pk2(__uint_as_float(x[i + 2]), __uint_as_float(x[i + 3])), mx::pk2(k4.z, k4.w),
                                    mx::mul2(qs2, mx::pk2(b4.z, b4.w)));
        float a, b;
        mx::upk2(mx::fma2(ra2, u, add_2), a, b);
        x[i] = __float_as_uint(a), x[i + 1] = __float_as_uint(b);
        mx::upk2(mx::fma2(ra2, w, add_2), a, b);
        x[i + 2] = __float_as_uint(a), x[i + 3] = __float_as_uint(b);
    }
}
// maximum of 64 scores: four independent chains (a single one would serialise on the latency)
__device__ __forceinline__ float fwd_max64(const uint32_t (&va)[32], const uint32_t (&vb)[32]) {
    float mx4[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) mx4[u] = fmaxf(__uint_as_float(va[u]), __uint_as_float(vb[u]));
#pragma unroll
    for (int i = 4; i < 32; i += 4)
#pragma unroll
        for (int u = 0; u < 4; ++u) mx4[u] = fmax3(mx4[u], __uint_as_float(va[i + u]), __uint_as_float(vb[i + u]));
    return fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
}
__device__ __forceinline__ void fwd_mask64(uint32_t (&va)[32], uint32_t (&vb)[32], int key_base, int last) {   // keys this row does not see
#pragma unroll
    for (int i = 0; i < 32; ++i) {
        if (key_base + i > last) va[i] = 0xFF800000u;  // -inf
        if (key_base + 32 + i > last) vb[i] = 0xFF800000u;
    }
}
// Max-free loop: 32 scores of a row -> probabilities, packed to bf16, and their sum (packed pairs; `start`: the first of a tile).
// nmc: minus the reference in log2 units (REF sources).  scores: src holds finished, masked scores.
template <int SRC>
__device__ __forceinline__ void fwd_exp32(const uint32_t *src, uint32_t *pk, int key_base, int last, bool need_mask, const float *kskb,
                                          bool start, bool scores, float nmc, float row_a, float row_qsum, uint64_t &rs2) {
    constexpr bool RAW = SRC == SRC_RAW || SRC == SRC_RAW_BOUND, REF = SRC != SRC_PRE;
    constexpr float c = RAW ? MX230_QK_LOG2_SCALE : 1.0f;
    constexpr int POLY = SRC == SRC_PRE ? FWD_POLY : 0;   // (the rebuilt int8 scores leave the exp unit time enough)
    uint32_t x[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) x[i] = src[i];
    if (RAW || (REF && scores)) {   // to log2 units, against the reference
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
            float a, b;
            mx::upk2(mx::fma2(mx::pk2(__uint_as_float(x[i]), __uint_as_float(x[i + 1])), mx::pk2(c, c), mx::pk2(nmc, nmc)), a, b);
            x[i] = __float_as_uint(a), x[i + 1] = __float_as_uint(b);
        }
    } else if (SRC == SRC_I8) {
        fwd_rebuild32(x, kskb, nmc, row_a, row_qsum);
    }
    if (need_mask && !scores) {   // diagonal and ragged tiles only (a warp-uniform branch: full tiles pay nothing)
#pragma unroll
        for (int i = 0; i < 32; ++i)
            if (key_base + i > last) x[i] = (POLY > 0) ? 0xC2FC0000u : 0xFF800000u;  // -126 (2^-126 against sums >= 2^-80) | -inf
    }
#pragma unroll
    for (int i = 0; i < 32; i += 2) {
        float p0, p1;
        if (((i >> 1) % FWD_POLY_DEN) < POLY) {
            mx::ex2_poly2<false>(__uint_as_float(x[i]), __uint_as_float(x[i + 1]), p0, p1);
        } else {
            p0 = mx::ex2(__uint_as_float(x[i]));
            p1 = mx::ex2(__uint_as_float(x[i + 1]));
        }
        pk[i >> 1] = mx::pack_bf16(p0, p1);
        rs2 = start && i == 0 ? mx::pk2(p0, p1) : mx::add2(rs2, mx::pk2(p0, p1));
    }
}

// KEY_SPLIT: an item is ONE query tile whose even key tiles belong to softmax groups 0, 1 and whose odd ones to groups 2, 3,
// each pair with its own S and P in tensor memory, so that both pairs of groups work on every item and items are half as
// large (fwd_key_split says when).  Without a row max P V of all key tiles is summed into one O in key order, and both
// forms sum a row's probabilities over even and odd key tiles apart: a head's result has the same bits in either form.
// With a row max each pair of groups has its own max and its own O, which the first group joins at the end.
// HALF: the output goes to O_half as well (an instantiation of its own: as a run-time choice it made the int8 key-split loop 3 to
// 5 % slower, 512 tokens over 2048 keys 28.4 -> 29.2 us).
template <int SRC, bool KEY_SPLIT, bool HALF>
__global__ void __launch_bounds__(FWD_THREADS, 1)
flash_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                 const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmO,
                 const FwdParams P) {
    extern __shared__ unsigned char smem_dyn[];
    const uint32_t smem_base = (mx::smem_u32(smem_dyn) + 1023u) & ~1023u;
    unsigned char *smem = smem_dyn + (smem_base - mx::smem_u32(smem_dyn));
    const uint32_t bar0 = smem_base + SMEM_BAR;
    auto bar = [&](int i) { return bar0 + 8u * (uint32_t)i; };
    volatile uint32_t *tmem_slot = (volatile uint32_t *)(smem + SMEM_BAR + 8 * N_BARS);
    volatile int *abort_flag = (volatile int *)(smem + SMEM_BAR + 8 * N_BARS + 8);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int NQ = P.n_q, N = P.n_k;  // N: keys (bounds the K/V loop and the key mask)

    if (tid == 0) {
        for (int b = 0; b < Q_BUFS; ++b) {
            mx::mbar_init(bar(BAR_Q_FULL + b), 1);
            mx::mbar_init(bar(BAR_Q_EMPTY + b), SOFT_WARPS);  // one elected lane per softmax warp arrives
        }
        for (int s = 0; s < KV_STAGES; ++s) {
            mx::mbar_init(bar(BAR_K_FULL + s), 1);
            mx::mbar_init(bar(BAR_K_EMPTY + s), 1);
            mx::mbar_init(bar(BAR_V_FULL + s), 1);
            mx::mbar_init(bar(BAR_V_EMPTY + s), 1);
        }
        for (int t = 0; t < QT; ++t) {
            mx::mbar_init(bar(BAR_S_FULL + t), 1);
            mx::mbar_init(bar(BAR_S_FREE + t), HALVES * BM / 32);  // one elected lane per warp of the tile's groups arrives
            mx::mbar_init(bar(BAR_P_FULL + t), HALVES * BM / 32);
            mx::mbar_init(bar(BAR_O_DONE + t), 1);
            mx::mbar_init(bar(BAR_XCH + t), (KEY_SPLIT ? XCH_PUBS : 1) * BM / 32);
            mx::mbar_init(bar(BAR_XMAX + t), HALVES * BM / 32);
        }
        mx::mbar_init(bar(BAR_O1_READ), BM / 32);
        *abort_flag = 0;
        mx::mbar_fence_init();
    }
    if (warp == SOFT_WARPS + 1) mx::tmem_alloc(mx::smem_u32((const void *)tmem_slot), TM_COLS);
    mx::tc_fence_before();
    __syncthreads();
    mx::tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    if (KEY_SPLIT) fwd_prefetch_maps(P, warp, lane, tmQ, tmK, tmV, tmO);
    // In the key-split form, which short calls take, every role waits for the previous kernel behind the arithmetic of its first
    // item: it took 0.4 us behind the wait (code and parameters come into the caches with it; 12 x 1024 rows causal 15.2 -> 14.7).
    // Not with int8 scores, whose loop comes out slower then (attention of 700 tokens over
    // 4700 keys, 14/2 heads, 46.6 us against 44.0; 14 such sizes 0 to 6 % slower).
    constexpr bool SHORT = KEY_SPLIT && SRC != SRC_I8;
    if (!SHORT) mx::pdl_wait();

    if (warp >= SOFT_WARPS) {
        if (warp == SOFT_WARPS) {
        // ------------------------- TMA producer -------------------------
        if (lane == 0) {
            if (!KEY_SPLIT) fwd_prefetch_maps(P, warp, lane, tmQ, tmK, tmV, tmO);
            bool ok = true;
            uint32_t g = 0;  // K/V tiles loaded so far, over all items: ring slot g % KV_STAGES, use g / KV_STAGES
            int bh, q0;
            for (int it = 0; ok && fwd_item(P, it, bh, q0); ++it) {
                const int n_it1 = KEY_SPLIT ? 0 : fwd_tile_iters(P, q0, 1);
                const int n_max = max(fwd_tile_iters(P, q0, 0), n_it1);
                const int qbuf = it & 1;
                // the buffer's previous item (two items ago) must have staged its last O piece out of it
                if (it >= Q_BUFS) ok = mx::mbar_wait(bar(BAR_Q_EMPTY + qbuf), ((it >> 1) - 1) & 1, abort_flag, P.status);
                if (!ok) break;
                const int nq = (n_it1 > 0) ? 2 : 1;
                if (SHORT && it == 0) mx::pdl_wait();
                mx::mbar_expect_tx(bar(BAR_Q_FULL + qbuf), nq * TILE_BYTES);
                for (int t = 0; t < nq; ++t)
                    mx::tma_load_3d(smem_base + SMEM_Q + (qbuf * QT + t) * TILE_BYTES, &tmQ, bar(BAR_Q_FULL + qbuf), 0,
                                    q0 + t * BM, bh);
                const int kvh = bh / P.kv_group;
                for (int j = 0; j < n_max; ++j, ++g) {
                    const int s = g % KV_STAGES;
                    const uint32_t r = g / KV_STAGES;
                    if (r > 0) ok = mx::mbar_wait(bar(BAR_K_EMPTY + s), (r - 1) & 1, abort_flag, P.status);
                    if (!ok) break;
                    if (P.test_drop_tile == (int)g && blockIdx.x == 0) continue;   // test hook: this tile never arrives
                    mx::mbar_expect_tx(bar(BAR_K_FULL + s), TILE_BYTES + (SRC == SRC_I8 ? KSKB_BYTES : 0));
                    mx::tma_load_3d(smem_base + SMEM_K + s * TILE_BYTES, &tmK, bar(BAR_K_FULL + s), 0,
                                    j * BN, kvh);
                    // The tile's scales and offsets land before its scores exist.  Slot g % 8 is free: this thread has
                    // loaded V of tile g - 1 before, over V of tile g - 5, so P V of every tile up to g - 5 is complete, and
                    // it waited for the probabilities of all warps that read the tile's scales (in both loops the last
                    // read comes before the arrival on P_FULL).  That holds in either form, whichever groups a tile has.
                    if (SRC == SRC_I8)
                        mx::bulk_load(smem_base + SMEM_KSKB + (g % KSKB_SLOTS) * KSKB_BYTES,
                                      P.col_kskb + ((size_t)kvh * P.n_k_tiles + j) * 2 * BN, KSKB_BYTES, bar(BAR_K_FULL + s));
                    if (r > 0) ok = mx::mbar_wait(bar(BAR_V_EMPTY + s), (r - 1) & 1, abort_flag, P.status);
                    if (!ok) break;
                    mx::mbar_expect_tx(bar(BAR_V_FULL + s), TILE_BYTES);
                    mx::tma_load_3d(smem_base + SMEM_V + s * TILE_BYTES, &tmV, bar(BAR_V_FULL + s), 0,
                                    j * BN, kvh);
                }
            }
        }
        __syncwarp();
        } else if (warp == SOFT_WARPS + 1) {
        // ------------------------- MMA issuer 1: S_t = Q_t K^T ----------
        // The whole warp runs the loop and the waits; one elected lane issues.  Control flow and descriptor
        // arithmetic stay warp-uniform that way (a lone thread inside a divergent branch pays several dependent
        // instructions per tcgen05.mma to move its operands to the uniform registers the instruction reads).
        {
            constexpr uint32_t IDESC_S = mx::mma_idesc_bf16(BM, BN, false, false);
            bool ok = true;
            uint32_t g = 0;            // K/V tiles consumed so far, over all items
            uint32_t cs[QT] = {0, 0};  // score tiles issued so far per query tile, over all items
            int bh, q0;
            for (int it = 0; ok && fwd_item(P, it, bh, q0); ++it) {
                int n_it[QT];
#pragma unroll
                for (int t = 0; t < QT; ++t) n_it[t] = fwd_tile_iters(P, q0, KEY_SPLIT ? 0 : t);
                const int n_max = max(n_it[0], n_it[1]);
                const int qbuf = it & 1;
                if (SHORT && it == 0) mx::pdl_wait();
                ok = ISSUER_WAIT(mx::mbar_wait(bar(BAR_Q_FULL + qbuf), (it >> 1) & 1, abort_flag, P.status));
                for (int j = 0; j < n_max && ok; ++j, ++g) {
                    const int s = g % KV_STAGES;
                    ok = ISSUER_WAIT(mx::mbar_wait(bar(BAR_K_FULL + s), (g / KV_STAGES) & 1, abort_flag, P.status));
                    const uint64_t b = mx::smem_desc_sw128(smem_base + SMEM_K + s * TILE_BYTES);
#pragma unroll
                    for (int t = 0; t < QT; ++t) {
                        if (!ok || j >= n_it[t] || (KEY_SPLIT && (j & 1) != t)) continue;
                        // next scores as soon as the softmax group holds the previous ones in registers (the
                        // previous ones may be the last of the item before: this is where the items overlap)
                        if (cs[t] > 0) ok = ISSUER_WAIT(mx::mbar_wait(bar(BAR_S_FREE + t), (cs[t] - 1) & 1, abort_flag, P.status));
                        if (!ok) continue;
                        mx::tc_fence_after();
                        const uint64_t a = mx::smem_desc_sw128(smem_base + SMEM_Q + (qbuf * QT + (KEY_SPLIT ? 0 : t)) * TILE_BYTES);
                        if (ISSUER_LANE) {
#pragma unroll
                            for (int k = 0; k < HD / 16; ++k)  // 32 bytes per 16-element step inside the swizzle span
                                mx::mma_ss(tmem + TM_S + t * BN, a + 2 * k, b + 2 * k, IDESC_S, k > 0);
                            mx::mma_commit(bar(BAR_S_FULL + t));
                        }
                        ++cs[t];
                    }
                    if (!ok) break;
                    if (ISSUER_LANE) mx::mma_commit(bar(BAR_K_EMPTY + s));
                }
            }
        }
        __syncwarp();
        } else if (warp == SOFT_WARPS + 2) {
        // ------------------------- MMA issuer 2: O_t += P_t V -----------
        {
            constexpr uint32_t IDESC_O = mx::mma_idesc_bf16(BM, HD, false, true);
            bool ok = true;
            uint32_t g = 0;            // K/V tiles consumed so far, over all items
            uint32_t cp[QT] = {0, 0};  // P tiles consumed so far per query tile, over all items
            int bh, q0;
            for (int it = 0; ok && fwd_item(P, it, bh, q0); ++it) {
                int n_it[QT];
#pragma unroll
                for (int t = 0; t < QT; ++t) n_it[t] = fwd_tile_iters(P, q0, KEY_SPLIT ? 0 : t);
                const int n_max = max(n_it[0], n_it[1]);
                if (SHORT && it == 0) mx::pdl_wait();
                // each pair of groups sums into an O of its own
                const bool own_o = !KEY_SPLIT || SRC == SRC_RAW ||
                                   !(SRC == SRC_RAW_BOUND
                                         ? fwd_fast_raw(P, bh, q0)
                                         : fwd_fast_head(P, bh, lane, SRC == SRC_I8 ? FAST_BOUND_REF : FAST_BOUND));
                for (int j = 0; j < n_max && ok; ++j, ++g) {
                    const int s = g % KV_STAGES;
                    ok = ISSUER_WAIT(mx::mbar_wait(bar(BAR_V_FULL + s), (g / KV_STAGES) & 1, abort_flag, P.status));
                    const uint64_t b = mx::smem_desc_sw128(smem_base + SMEM_V + s * TILE_BYTES);
#pragma unroll
                    for (int t = 0; t < QT; ++t) {
                        if (!ok || j >= n_it[t] || (KEY_SPLIT && (j & 1) != t)) continue;
                        // an item's first P_t is written after the softmax group has taken the previous item's
                        // O_t out of tensor memory, so overwriting O_t (j == 0) needs no barrier of its own
                        ok = ISSUER_WAIT(mx::mbar_wait(bar(BAR_P_FULL + t), cp[t] & 1, abort_flag, P.status));
                        if (!ok) continue;
                        mx::tc_fence_after();
                        if (ISSUER_LANE) {
#pragma unroll
                            for (int k = 0; k < BN / 16; ++k)  // 16 keys: 8 packed columns of P, 2048 bytes of V
                                mx::mma_ts(tmem + TM_O + (own_o ? t * HD : 0), tmem + TM_P + t * (BN / 2) + 8 * k, b + 128 * k,
                                           IDESC_O, (j > (KEY_SPLIT && own_o ? t : 0) || k > 0));
                            mx::mma_commit(bar(BAR_O_DONE + t));
                        }
                        ++cp[t];
                    }
                    if (!ok) break;
                    if (ISSUER_LANE) mx::mma_commit(bar(BAR_V_EMPTY + s));
                }
            }
        }
        __syncwarp();
        }
    } else {
        // ------------------------- softmax groups -----------------------
        // Four groups: tile t = warp / 8 has two, each taking 64 of the 128 key columns of every score tile (one thread
        // per query row and half).  Four softmax warps per scheduler instead of two hide each other's dependent-issue
        // latencies; without a row max (the usual mode) the halves never talk to each other inside the loop, and the
        // general mode has them exchange their part of the row max per score tile.
        const int t = warp >> 3;             // query tile of this group (key-split form: parity of its key tiles)
        const int half = (warp >> 2) & 1;    // which 64 key columns of every tile
        const int row_in_tile = (warp & 3) * 32 + lane;
        const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
        const uint32_t tm_s_tile = tmem + lane_off + TM_S + t * BN;
        const uint32_t tm_s = tm_s_tile + half * (BN / 2);
        const uint32_t tm_p = tmem + lane_off + TM_P + t * (BN / 2) + half * (BN / 4);
        const uint32_t tm_o = tmem + lane_off + TM_O + t * HD;
        // Scores arrive in log2 units when Q was staged pre-multiplied by scale * log2(e) or when they are rebuilt from
        // integer dots (c = 1), else raw (c = scale * log2(e)).
        constexpr bool RAW = SRC == SRC_RAW || SRC == SRC_RAW_BOUND;
        constexpr float c = RAW ? MX230_QK_LOG2_SCALE : 1.0f;
        constexpr float l_scale = RAW ? 0.125f : 0.6931471805599453f;   // running max -> natural-log units
        // These sources need a multiply per score anyway, which subtracts a reference for free: the max-free loop then takes
        // probabilities against the row's max over the first key tile, as the general loop does until a later tile raises
        // it (against 0 the leading probability is rounded like any other: 1 to 8 % more error with int8 scores).
        constexpr bool REF = SRC != SRC_PRE;
        bool ok = true;
        uint32_t cnt = 0;  // score tiles this group has taken so far, over all items
        uint32_t cnt1 = 0; // key-split form: odd key tiles so far (what groups 2, 3 count in cnt)
        uint32_t g0 = 0;   // key tiles of the items so far (int8 scores: ring position)
        uint32_t xmc = 0;  // row-max exchanges this tile's groups have made so far
        uint32_t xmc0 = 0; // key-split form, odd groups: those of the even ones
        uint32_t turn = 0; // items this tile's groups have worked on
        int bh, q0;
        for (int it = 0; ok && fwd_item(P, it, bh, q0); ++it) {
        const int n_all = KEY_SPLIT ? fwd_tile_iters(P, q0, 0) : 0;
        const int n_t = KEY_SPLIT ? (n_all + 1 - t) >> 1 : fwd_tile_iters(P, q0, t);
        const int row0 = q0 + (KEY_SPLIT ? 0 : t * BM);   // first row of this group's query tile
        const int row = row0 + row_in_tile;
        const int qbuf = it & 1;
        // Pair form, the last rows of a head with an odd number of query tiles: there is no second tile, and its groups pass
        // the item over; the first tile's arrive on the Q buffer's barrier in their place.  (Taking part without any work,
        // they would run ahead of the first tile from one such item to the next, and a barrier that counts one item's
        // arrivals cannot tell them from the next but one's.)
        const bool lone = !KEY_SPLIT && q0 + BM >= NQ;
        if (SHORT && it == 0) mx::pdl_wait();
        if (lone && t == 1) {
            g0 += fwd_tile_iters(P, q0, 0);
            continue;
        }
        auto key_tile = [&](int j) { return KEY_SPLIT ? 2 * j + t : j; };
        float row_a = 0.0f, row_qsum = 0.0f;
        if (SRC == SRC_I8 && row < NQ) {
            row_a = P.row_a[(size_t)bh * NQ + row];
            row_qsum = P.row_qsum[(size_t)bh * NQ + row];
        }
        // int8 scores: ks (and BN floats further kb) of this half's columns of the group's j-th key tile
        auto kskb_of = [&](int j) {
            return (const float *)(smem + SMEM_KSKB + ((g0 + (uint32_t)key_tile(j)) % KSKB_SLOTS) * KSKB_BYTES) + half * (BN / 2);
        };
        // key-split form: O_1 of the previous item has been read (asked once per item by both halves of tile 1, so that
        // they stay in step with the reader)
        auto o1_free = [&]() {
            if (KEY_SPLIT && t == 1 && it > 0)
                return (bool)__all_sync(0xFFFFFFFFu, mx::mbar_wait(bar(BAR_O1_READ), (it - 1) & 1, abort_flag, P.status));
            return true;
        };
        const int last = P.causal ? min(N - 1, row + P.q_off) : N - 1;  // last visible key of this row
        // Fixed-reference mode, chosen per head: when |q . k| * scale * log2(e) is bounded for every row pair of the head --
        // by Cauchy-Schwarz from the largest row norms of Q and K -- the probabilities are taken against a reference that
        // stays: no running max, no rescale of O.  Q staged in log2 units (SRC_PRE): bound 80, reference 0, not even a
        // subtraction.  int8 scores and bounded bf16 operands (REF): bound 40, reference the row's max over its first key
        // tile.  Either way a probability is at most 2^80; bf16 probabilities and fp32 sums carry the same relative
        // precision at 2^-80 .. 2^80 as around 1, every row sum stays inside [2^-80, N 2^80], and the result is that of the
        // max-subtracted form.  Heads with larger scores (and calls without a bound) take the general path: running max,
        // lazy rescale.
        const bool fast = SRC == SRC_RAW ? false
                          : SRC == SRC_RAW_BOUND ? fwd_fast_raw(P, bh, row0)
                                                 : fwd_fast_head(P, bh, lane, REF ? FAST_BOUND_REF : FAST_BOUND);
        float m = fast ? 0.0f : -CUDART_INF_F, l = 0.0f;   // l: this group's share of the row sum
        float l_odd = 0.0f;    // pair form, fast mode: the sum over odd key tiles, l being that over even ones
        // Shares of the row sums, handed to the group that does the epilogue: [publisher][sum, second sum or max, correction].
        // The correction (what the first key tile's rounding adds to the sum that O is divided by: fast mode, see below) is
        // parked there from the first tile on, by the groups that publish nothing as well, instead of in a register.
        // (addresses are formed where they are used: pointers kept over the loop cost registers it needs)
        auto xch = [&](int pub, int what) -> float & {
            return ((float *)(smem + SMEM_XCH))[(((turn & 1) * XCH_PUBS + pub) * 3 + what) * BM + row_in_tile];
        };
        const int my_pub = KEY_SPLIT ? 2 * t + half - 1 : t;
        auto park = [&]() -> float & {
            return half == 1 || (KEY_SPLIT && t == 1) ? xch(my_pub, 2) : xch(2, KEY_SPLIT ? 2 : t);
        };
        uint32_t va[32], vb[32];
        auto rebuild32 = [&](uint32_t *x, const float *kskb, float add) { fwd_rebuild32(x, kskb, add, row_a, row_qsum); };
        // the halves of a row exchange their maxima of one score tile through shared memory (one bounded barrier)
        float *xmax = (float *)(smem + SMEM_XMAX) + row_in_tile;   // [QT][2 exchange parities][HALVES][BM]
        auto row_max = [&](float own) -> float {
            float *xm = xmax + (t * 2 + (xmc & 1)) * HALVES * BM;
            xm[half * BM] = own;
            __syncwarp();
            if (lane == 0) mx::mbar_arrive(bar(BAR_XMAX + t));
            ok = __all_sync(0xFFFFFFFFu, mx::mbar_wait(bar(BAR_XMAX + t), xmc & 1, abort_flag, P.status));
            ++xmc;
            return fmaxf(own, xm[(1 - half) * BM]);
        };
        auto max64 = [&]() { return fwd_max64(va, vb); };
        auto mask64 = [&](int key_base) { fwd_mask64(va, vb, key_base, last); };
        if (fast) {
        float nmc = 0.0f;   // REF: minus the reference, in log2 units
        // ---- max-free loop: the group's second 32 columns land under the exponentials of the first 32
        uint64_t rs2;              // sum of one score tile
        float l_other = 0.0f;      // pair form: l and l_other change places after every tile: sums over even and odd key tiles
        auto exp32 = [&](const uint32_t *src, uint32_t *pk, int key_base, bool need_mask, const float *kskb, bool start, bool scores) {
            fwd_exp32<SRC>(src, pk, key_base, last, need_mask, kskb, start, scores, nmc, row_a, row_qsum, rs2);
        };
        // First key tile only: the sum of the ROUNDED probabilities as well.  Rows that see a handful of keys live
        // there (the first rows of a causal head), and for them the output has to be normalised by what the tensor
        // core actually multiplies with V -- a row with one visible key must return that row of V, not V times
        // bf16(p) / p, or dO . O stops cancelling against dP in the backward.  Everywhere else a row sums so many
        // terms that the two sums differ far below the rounding of V itself, and the fp32 sum serves both uses.
        float rb[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        auto sum_rounded16 = [&](const uint32_t *pk) {
#pragma unroll
            for (int w = 0; w < 16; ++w) mx::add_bf16x2(pk[w], rb[(w & 1) * 2], rb[(w & 1) * 2 + 1]);
        };
        auto sum_of = [](uint64_t v) {
            float a0, a1;
            mx::upk2(v, a0, a1);
            return a0 + a1;
        };
        // one score tile; FIRST (a compile-time flag: the loop below stays free of the first tile's extra work) also
        // takes the sums of the rounded probabilities
        auto tile = [&](auto first_c, int j) -> bool {
            constexpr bool FIRST = decltype(first_c)::value;
            bool good = __all_sync(0xFFFFFFFFu, mx::mbar_wait(bar(BAR_S_FULL + t), cnt & 1, abort_flag, P.status));
            if (!good) return false;
            mx::tc_fence_after();
            mx::tmem_ld32(tm_s, va);
            mx::tmem_wait_ld();                                       // va is in registers
            mx::tmem_ld32(tm_s + 32, vb);                             // lands under the first exponentials
            const int key0 = key_tile(j) * BN;
            const bool need_mask = (key0 + BN > N) || (P.causal && key0 + BN - 1 > row0 + P.q_off);
            const float *kskb = SRC == SRC_I8 ? kskb_of(j) : nullptr;
            uint32_t pk[16];
            constexpr bool LEAD = REF && FIRST;
            const bool scores = LEAD && !(KEY_SPLIT && t == 1);   // va, vb hold masked scores already
            if (scores) {   // the reference: the row's max over its first key tile
                mx::tmem_wait_ld();
                if (SRC == SRC_I8) rebuild32(va, kskb, 0.0f), rebuild32(vb, kskb + 32, 0.0f);
                if (need_mask) mask64(key0 + half * (BN / 2));
                m = row_max(max64());
                if (!ok) return false;
            } else if (LEAD) {   // odd key tiles of the key-split form: that of the even ones
                good = __all_sync(0xFFFFFFFFu, mx::mbar_wait(bar(BAR_XMAX), xmc0 & 1, abort_flag, P.status));
                if (!good) return false;
                const float *xm = xmax + (xmc0 & 1) * HALVES * BM;
                m = fmaxf(xm[0], xm[BM]);
            }
            if (LEAD) nmc = -m * c;
            exp32(va, pk, key0 + half * (BN / 2), need_mask, kskb, true, scores);
            mx::tmem_wait_ld();                                       // this group's columns have left S_t
            mx::tc_fence_before();
            __syncwarp();
            if (lane == 0) mx::mbar_arrive(bar(BAR_S_FREE + t));
            if (!FIRST) {
                // P_t is free once the previous P V has completed: that takes several hundred cycles from the end of the
                // previous softmax, which is why a quarter of the row is exponentiated before the first store
                good = __all_sync(0xFFFFFFFFu,
                                  mx::mbar_wait_fast(bar(BAR_O_DONE + t), (cnt - 1) & 1, abort_flag, P.status));
                if (!good) return false;
                mx::tc_fence_after();
            }
            mx::tmem_st16(tm_p, pk);
            if (FIRST && !(KEY_SPLIT && t == 1)) sum_rounded16(pk);
            exp32(vb, pk, key0 + half * (BN / 2) + 32, need_mask, kskb + 32, false, scores);
            mx::tmem_st16(tm_p + 16, pk);
            if (FIRST) {
                if (!(KEY_SPLIT && t == 1)) {
                    sum_rounded16(pk);
                    park() = ((rb[0] + rb[1]) + (rb[2] + rb[3])) - sum_of(rs2);
                }
                if (!o1_free()) return false;
            }
            mx::tmem_wait_st();
            mx::tc_fence_before();
            __syncwarp();
            if (lane == 0) mx::mbar_arrive(bar(BAR_P_FULL + t));
            const float l_new = l + sum_of(rs2);
            if (KEY_SPLIT) {
                l = l_new;
            } else {   // the next key tile has the other parity
                l = l_other;
                l_other = l_new;
            }
            return true;
        };
        if (n_t > 0) {
            ok = tile(std::true_type{}, 0);
            ++cnt;
            for (int j = 1; ok && j < n_t; ++j) {
                ok = tile(std::false_type{}, j);
                ++cnt;
            }
        }
        if (!KEY_SPLIT) {
            l_odd = (n_t & 1) ? l : l_other;
            if (n_t & 1) l = l_other;
        }
        } else {
        // ---- general loop: running row max, raised lazily.  Each half takes the max of its own 64 columns and the two
        // exchange them through shared memory (one bounded barrier per tile and query tile); both then hold the same
        // row max and take the same decisions, exponentiate their own columns and rescale their own 32 columns of O.
        for (int j = 0; j < n_t; ++j, ++cnt) {
            ok = __all_sync(0xFFFFFFFFu, mx::mbar_wait(bar(BAR_S_FULL + t), cnt & 1, abort_flag, P.status));
            if (!ok) break;
            mx::tc_fence_after();
            mx::tmem_ld32(tm_s, va);
            mx::tmem_ld32(tm_s + 32, vb);
            mx::tmem_wait_ld();
            mx::tc_fence_before();
            __syncwarp();
            if (lane == 0) mx::mbar_arrive(bar(BAR_S_FREE + t));   // this group's columns have left S_t
            const int key0 = key_tile(j) * BN, col0 = half * (BN / 2);
            if (SRC == SRC_I8) {   // the tile holds exact integer dots of int8 codes: the reference kernel's score for them
                const float *kskb = kskb_of(j);
                rebuild32(va, kskb, 0.0f);
                rebuild32(vb, kskb + 32, 0.0f);
            }
            if ((key0 + BN > N) || (P.causal && key0 + BN - 1 > row0 + P.q_off)) mask64(key0 + col0);
            const float mx_ = row_max(max64());
            if (!ok) break;
            // raise the running max only when it pays (always on the first tile)
            const bool raise = (j == 0) || ((mx_ - m) * c > RESCALE_LOG2);
            const float m_new = raise ? mx_ : m;
            const float alpha = (raise && j > 0) ? mx::ex2((m - m_new) * c) : 1.0f;
            // (key-split form: a row may see none of the group's first key tiles; its max is still -inf then)
            const float nmc = KEY_SPLIT && m_new == -CUDART_INF_F ? 0.0f : -m_new * c;
            if (j > 0) {
                // P_t and O_t are stable once the previous P V has completed
                ok = __all_sync(0xFFFFFFFFu,
                                mx::mbar_wait(bar(BAR_O_DONE + t), (cnt - 1) & 1, abort_flag, P.status));
                if (!ok) break;
                mx::tc_fence_after();
                if (__any_sync(0xFFFFFFFFu, raise)) {
#pragma unroll 1
                    for (int cc = 0; cc < 2; ++cc) {
                        uint32_t o[16];
                        mx::tmem_ld16(tm_o + half * 32 + cc * 16, o);
                        mx::tmem_wait_ld();
#pragma unroll
                        for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
                        mx::tmem_st16(tm_o + half * 32 + cc * 16, o);
                    }
                }
            }
            float rs[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            uint32_t pk[16];
#pragma unroll
            for (int i = 0; i < 32; i += 2) {
                const float p0 = mx::ex2(fmaf(__uint_as_float(va[i]), c, nmc));
                const float p1 = mx::ex2(fmaf(__uint_as_float(va[i + 1]), c, nmc));
                rs[i & 2] += p0;
                rs[(i & 2) + 1] += p1;
                pk[i >> 1] = mx::pack_bf16(p0, p1);
            }
            mx::tmem_st16(tm_p, pk);
#pragma unroll
            for (int i = 0; i < 32; i += 2) {
                const float p0 = mx::ex2(fmaf(__uint_as_float(vb[i]), c, nmc));
                const float p1 = mx::ex2(fmaf(__uint_as_float(vb[i + 1]), c, nmc));
                rs[i & 2] += p0;
                rs[(i & 2) + 1] += p1;
                pk[i >> 1] = mx::pack_bf16(p0, p1);
            }
            mx::tmem_st16(tm_p + 16, pk);
            l = l * alpha + ((rs[0] + rs[1]) + (rs[2] + rs[3]));
            m = m_new;
            if (KEY_SPLIT && j == 0) {
                ok = o1_free();
                if (!ok) break;
            }
            mx::tmem_wait_st();
            mx::tc_fence_before();
            __syncwarp();
            if (lane == 0) mx::mbar_arrive(bar(BAR_P_FULL + t));
        }
        }
        if (KEY_SPLIT && n_t == 0 && ok) ok = o1_free();
        // The groups of a row add their sums: half 1 (key-split form: every group but the first) publishes its share and
        // goes on to the next item; the first group waits for it, and for the last P V, and does the tile's epilogue.
        float l_norm = 0.0f;             // what O is divided by
        float w0 = 1.0f, w1 = 1.0f;      // key-split form, general mode: weights of O_0 and O_1
        if (half == 1 || (KEY_SPLIT && t == 1)) {
            // The odd groups of the key-split form publish before their last P V is complete, so that the first group has their sums
            // when it is.  None publishes twice before the first group has taken the first: O1_READ, which they wait for in every
            // item, comes behind that.  (The others publish behind an item's last P V, which the first group's P precedes: with no
            // such order a second arrival could pass for one that is missing.  The other sources' odd groups wait for an exchange
            // first, below.)
            const bool early = KEY_SPLIT && (SRC == SRC_PRE || SRC == SRC_RAW) && t == 1;
            if (early && ok) {
                xch(my_pub, 0) = l;
                xch(my_pub, 1) = m;
                __syncwarp();
                if (lane == 0) mx::mbar_arrive(bar(BAR_XCH));
            }
            // (the tile's last P V must have read this group's share of P_t before the next item's first tile overwrites it)
            if (ok && n_t > 0)
                ok = __all_sync(0xFFFFFFFFu, mx::mbar_wait(bar(BAR_O_DONE + t), (cnt - 1) & 1, abort_flag, P.status));
            // Key-split form, sources whose max-free loop takes its reference from the even groups' exchange: the odd groups
            // see every item's last exchange complete before they go on, also where they take nothing from it.  A parity
            // wait tells a phase from the one before, not from the one before that: with an exchange still open, the next
            // item's wait would return on an older one and read another head's maxima.  (The exchange before the last is
            // behind the P V that was waited for above, and none can follow the last before these groups have published.)
            if (KEY_SPLIT && t == 1 && (SRC == SRC_RAW_BOUND || SRC == SRC_I8)) {
                xmc0 += fast ? 1u : (uint32_t)((n_all + 1) >> 1);
                if (ok) ok = __all_sync(0xFFFFFFFFu, mx::mbar_wait(bar(BAR_XMAX), (xmc0 - 1) & 1, abort_flag, P.status));
            }
            if (ok && !early) {
                xch(my_pub, 0) = l;
                xch(my_pub, 1) = KEY_SPLIT ? m : l_odd;
                __syncwarp();
                if (lane == 0) mx::mbar_arrive(bar(BAR_XCH + (KEY_SPLIT ? 0 : t)));
            }
        } else if (ok) {
            ok = __all_sync(0xFFFFFFFFu, mx::mbar_wait(bar(BAR_XCH + t), turn & 1, abort_flag, P.status));
            if (ok) {
                const int other = KEY_SPLIT ? 0 : t;   // half 1 of this tile
                l += xch(other, 0);
                const float corr = fast ? park() + xch(other, 2) : 0.0f;
                if (KEY_SPLIT) {
                    l_odd = xch(1, 0) + xch(2, 0);
                    if (!fast) {
                        const float m1 = xch(1, 1), mm = fmaxf(m, m1);
                        w0 = mx::ex2((m - mm) * c);   // m is finite: key tile 0 has a key that every row sees
                        w1 = mx::ex2((m1 - mm) * c);
                        l *= w0, l_odd *= w1;
                        m = mm;
                    }
                } else {
                    l_odd += xch(other, 1);
                }
                l += l_odd;
                l_norm = l + corr;
            }
        }
        if (KEY_SPLIT) cnt1 += (uint32_t)(n_all >> 1);
        // epilogue: O / l and the log-sum-exp
        if (ok && n_t > 0 && half == 0 && !(KEY_SPLIT && t == 1)) {
            const bool odd = KEY_SPLIT && n_all > 1, two = odd && !fast;   // O_1 holds something
            ok = __all_sync(0xFFFFFFFFu,
                            mx::mbar_wait(bar(BAR_O_DONE + t), (cnt - 1) & 1, abort_flag, P.status));
            if (ok && odd) ok = __all_sync(0xFFFFFFFFu, mx::mbar_wait(bar(BAR_O_DONE + 1), (cnt1 - 1) & 1, abort_flag, P.status));
            if (ok) {
                mx::tc_fence_after();
                const float inv = 1.0f / l_norm;
                auto load_o = [&](int cc) {   // 32 columns of the row's sum into va
                    mx::tmem_ld32(tm_o + cc * 32, va);
                    if (two) mx::tmem_ld32(tm_o + HD + cc * 32, vb);
                    mx::tmem_wait_ld();
                    if (two) {
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                            va[i] = __float_as_uint(__uint_as_float(va[i]) * w0 + __uint_as_float(vb[i]) * w1);
                    }
                    if (KEY_SPLIT && cc == HD / 32 - 1) {   // O_1 has been read: the odd groups may go on to the next item
                        mx::tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mx::mbar_arrive(bar(BAR_O1_READ));
                    }
                };
                auto store_half = [&](int cc) {   // this row's 32 columns of va: 64 bytes
                    if (!HALF || row >= NQ) return;
                    uint4 *dst = (uint4 *)(P.O_half + ((size_t)bh * NQ + row) * HD + cc * 32);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        __half2 h2[4];
#pragma unroll
                        for (int u = 0; u < 4; ++u)
                            h2[u] = __floats2half2_rn(__uint_as_float(va[8 * i + 2 * u]) * inv, __uint_as_float(va[8 * i + 2 * u + 1]) * inv);
                        dst[i] = *(const uint4 *)h2;
                    }
                };
                float *orow = P.O + (size_t)bh * P.o_head_stride + (size_t)row * P.o_row_stride;
                if (P.tma_out) {
                    // each warp stages its 32 rows, 32 columns at a time, in a swizzled 4 KB piece of this tile's Q
                    // buffer (its last Q K^T has completed) and hands it to the TMA unit, which clips rows past the
                    // end: 16-byte stores from lane = row registers each touch a sector of their own
                    const int wrow0 = row0 + (warp & 3) * 32;
                    // (key-split form: in two such pieces, the item's second Q tile having no rows)
                    int st_off = SMEM_Q + (qbuf * QT + (KEY_SPLIT ? 0 : t)) * TILE_BYTES + (warp & 3) * 4096;
#pragma unroll 1
                    for (int cc = 0; cc < HD / 32; ++cc) {
                        if (SHORT && cc > 0) st_off += TILE_BYTES;
                        load_o(cc);
                        unsigned char *srow = smem + st_off + lane * 128;
#pragma unroll
                        for (int cch = 0; cch < 8; ++cch)
                            *(float4 *)(srow + ((cch ^ (lane & 7)) << 4)) =
                                make_float4(__uint_as_float(va[4 * cch]) * inv, __uint_as_float(va[4 * cch + 1]) * inv,
                                            __uint_as_float(va[4 * cch + 2]) * inv, __uint_as_float(va[4 * cch + 3]) * inv);
                        store_half(cc);
                        mx::fence_proxy_async_smem();
                        __syncwarp();
                        if (lane == 0 && wrow0 < NQ) {
                            mx::tma_store_3d(&tmO, smem_base + st_off, cc * 32, wrow0, bh);
                            mx::bulk_commit_group();
                            if (!SHORT || cc > 0) mx::bulk_wait_group_read<0>();   // the piece is reused and must outlive the read
                        }
                        __syncwarp();
                    }
                } else
#pragma unroll 1
                for (int cc = 0; cc < HD / 32; ++cc) {
                    load_o(cc);
                    if (row < NQ) {
#pragma unroll
                        for (int i = 0; i < 32; i += 4) {
                            float4 o4 = make_float4(__uint_as_float(va[i]) * inv, __uint_as_float(va[i + 1]) * inv,
                                                    __uint_as_float(va[i + 2]) * inv, __uint_as_float(va[i + 3]) * inv);
                            *(float4 *)(orow + cc * 32 + i) = o4;
                        }
                        store_half(cc);
                    }
                }
                if (P.L != nullptr && row < NQ) P.L[(size_t)bh * NQ + row] = m * l_scale + __logf(l);
            }
        }
        // this warp no longer touches the item's Q buffer (operand of its tile's Q K^T, then staging space)
        __syncwarp();
        if (ok && lane == 0) {
            mx::mbar_arrive(bar(BAR_Q_EMPTY + qbuf));
            if (lone) mx::mbar_arrive(bar(BAR_Q_EMPTY + qbuf));
        }
        ++turn;
        g0 += KEY_SPLIT ? n_all : max(fwd_tile_iters(P, q0, 0), fwd_tile_iters(P, q0, 1));
        }  // items
    }

    // ------------------------- teardown ---------------------------------
    mx::tc_fence_before();
    __syncthreads();
    mx::tc_fence_after();
    // The next kernel may move in from here on, when every warp is done.  Not earlier: what follows a long kernel would
    // fill the SMs that finish first with all of its blocks and find them unevenly spread when it may start (48 x 4096
    // rows, next call's cast: 9 us slower with the trigger at the top).
    mx::pdl_trigger();
    if (warp == SOFT_WARPS + 1) mx::tmem_dealloc(tmem, TM_COLS);
}

// ---- few items: 64 query rows each, the key tiles dealt to the four softmax groups in turn ----
// The same computation for calls whose 128-row items would leave SMs idle: a CTA has one item, 64 query rows, half the work of a
// key-split item, and its score tiles j, j + 1, j + 2, j + 3 are worked on at a time, one by each softmax group.  The tensor core
// computes 64 x 128 tiles (tcgen05.mma.ws), whose accumulators use all 128 lanes: lane l holds row l % 64, key columns
// 64 (l / 64) .., so that a thread has, as in the other forms, one row and 64 key columns, and everything a row sums up it sums
// up in the same order: P V of the key tiles into one O in key order, probabilities over even and odd key tiles apart.  A
// head's bits are those of the other forms (heads beyond the bound, whose groups each have a max and an O of their own, aside).
// P goes through shared memory (its lanes are not those that the tensor core would read it from).
// One item is the kernel's premise, not a loop's first turn: Q, the reference and the sums have one buffer, and a group's tile counts
// are its barriers' phases.  (With a loop over items, which no call ever took a second time, int8 scores spilled 252 bytes,
// staged fp32 92; 136 and 40 so.)
constexpr int R_ROWS = 64, R_GROUPS = 4, R_KS = 3, R_VS = 4;
constexpr int R_Q_BYTES = R_ROWS * HD * 2, R_P_BYTES = R_ROWS * BN * 2;   // P: two [64 rows][64 keys] swizzled tiles
constexpr int R_SLOTS = 4;
constexpr int R_SMEM_Q = 0;
constexpr int R_SMEM_K = R_SMEM_Q + R_Q_BYTES;
constexpr int R_SMEM_V = R_SMEM_K + R_KS * TILE_BYTES;
constexpr int R_SMEM_P = R_SMEM_V + R_VS * TILE_BYTES;
constexpr int R_SMEM_BAR = R_SMEM_P + R_GROUPS * R_P_BYTES;
constexpr int R_SMEM_KSKB = R_SMEM_BAR + 512;
constexpr int R_SMEM_SUM = R_SMEM_KSKB + KSKB_SLOTS * KSKB_BYTES;   // [groups 1..3][R_SLOTS][2][128] floats: what a group hands on with a tile
constexpr int R_SMEM_XMAX = R_SMEM_SUM + (R_GROUPS - 1) * R_SLOTS * 2 * 128 * 4;   // [groups][2][128] floats: row maxima of the halves
constexpr int R_SMEM_REF = R_SMEM_XMAX + R_GROUPS * 2 * 128 * 4;    // [64] floats: reference of the max-free loop
constexpr int R_SMEM_END = R_SMEM_REF + R_ROWS * 4;                 // [3][128] floats: sums of the halves
constexpr int R_ALLOC = R_SMEM_END + 3 * 128 * 4 + 1024;
static_assert(R_ALLOC <= 227 * 1024, "shared memory per CTA");
constexpr int RB_Q_FULL = 0, RB_K_FULL = RB_Q_FULL + 1, RB_K_EMPTY = RB_K_FULL + R_KS, RB_V_FULL = RB_K_EMPTY + R_KS,
              RB_V_EMPTY = RB_V_FULL + R_VS, RB_S_FULL = RB_V_EMPTY + R_VS, RB_S_FREE = RB_S_FULL + R_GROUPS,
              RB_P_FULL = RB_S_FREE + R_GROUPS, RB_P_DONE = RB_P_FULL + R_GROUPS, RB_XMAX = RB_P_DONE + R_GROUPS,
              RB_REF = RB_XMAX + R_GROUPS, RB_END = RB_REF + 1, R_BARS = RB_END + 1;
static_assert(8 * R_BARS + 16 <= 512, "barrier area");
constexpr int R_TM_S = 0, R_TM_O = R_GROUPS * (BN / 2);   // S of group w at w * 64, O of group w (max-free: one O, the first) at 256 + w * 32

template <int SRC, bool HALF>
__global__ void __launch_bounds__(FWD_THREADS, 1)
flash_fwd_rows64_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                        const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmO, const FwdParams P) {
    extern __shared__ unsigned char smem_dyn[];
    const uint32_t smem_base = (mx::smem_u32(smem_dyn) + 1023u) & ~1023u;
    unsigned char *smem = smem_dyn + (smem_base - mx::smem_u32(smem_dyn));
    const uint32_t bar0 = smem_base + R_SMEM_BAR;
    auto bar = [&](int i) { return bar0 + 8u * (uint32_t)i; };
    volatile uint32_t *tmem_slot = (volatile uint32_t *)(smem + R_SMEM_BAR + 8 * R_BARS);
    volatile int *abort_flag = (volatile int *)(smem + R_SMEM_BAR + 8 * R_BARS + 8);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int NQ = P.n_q, N = P.n_k;
    constexpr bool RAW = SRC == SRC_RAW || SRC == SRC_RAW_BOUND;
    constexpr bool REF = SRC != SRC_PRE;   // (see flash_fwd_kernel)
    constexpr float c = RAW ? MX230_QK_LOG2_SCALE : 1.0f;
    constexpr float l_scale = RAW ? 0.125f : 0.6931471805599453f;

    if (tid == 0) {
        for (int i = 0; i < R_BARS; ++i) {
            const bool by_warps = (i >= RB_S_FREE && i < RB_P_DONE) || i >= RB_XMAX;   // one elected lane of each of a group's warps
            mx::mbar_init(bar(i), by_warps ? 4 : 1);
        }
        *abort_flag = 0;
        mx::mbar_fence_init();
    }
    if (warp == SOFT_WARPS + 1) mx::tmem_alloc(mx::smem_u32((const void *)tmem_slot), TM_COLS);
    mx::tc_fence_before();
    __syncthreads();
    mx::tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    fwd_prefetch_maps(P, warp, lane, tmQ, tmK, tmV, tmO);

    // the item, heaviest first; n: key tiles that its rows see
    const int rank = blockIdx.x / P.heads, bh = blockIdx.x - rank * P.heads;
    const int q0 = (P.causal ? P.n_qblocks - 1 - rank : rank) * R_ROWS;
    const int n = P.causal ? min((N + BN - 1) / BN, (q0 + R_ROWS - 1 + P.q_off) / BN + 1) : (N + BN - 1) / BN;
    auto wait = [&](int b, uint32_t phase) { return mx::mbar_wait(bar(b), phase & 1, abort_flag, P.status); };
    auto wait_warp = [&](int b, uint32_t phase) { return (bool)__all_sync(0xFFFFFFFFu, wait(b, phase)); };
    auto head_fast = [&]() {
        return SRC == SRC_RAW ? false : SRC == SRC_RAW_BOUND ? fwd_fast_raw(P, bh, q0) : fwd_fast_head(P, bh, lane, REF ? FAST_BOUND_REF : FAST_BOUND);
    };
    bool ok = true;   // (every role waits for the previous kernel behind its own arithmetic, as in flash_fwd_kernel)
    if (warp == SOFT_WARPS) {
        // ------------------------- TMA producer -------------------------
        if (lane == 0) {
            const int kvh = bh / P.kv_group;
            mx::pdl_wait();
            mx::mbar_expect_tx(bar(RB_Q_FULL), R_Q_BYTES);
            mx::tma_load_3d(smem_base + R_SMEM_Q, &tmQ, bar(RB_Q_FULL), 0, q0, bh);
            for (int j = 0; j < n; ++j) {
                const int sk = j % R_KS, sv = j % R_VS;
                if (j >= R_KS) ok = wait(RB_K_EMPTY + sk, j / R_KS - 1);
                if (!ok) break;
                if (P.test_drop_tile == j && blockIdx.x == 0) continue;   // test hook: this tile never arrives
                mx::mbar_expect_tx(bar(RB_K_FULL + sk), TILE_BYTES + (SRC == SRC_I8 ? KSKB_BYTES : 0));
                mx::tma_load_3d(smem_base + R_SMEM_K + sk * TILE_BYTES, &tmK, bar(RB_K_FULL + sk), 0, j * BN, kvh);
                // (the slot of the scales of tile j - 8 is free: P V of every tile up to j - 5 is complete, see flash_fwd_kernel)
                if (SRC == SRC_I8)
                    mx::bulk_load(smem_base + R_SMEM_KSKB + (j % KSKB_SLOTS) * KSKB_BYTES,
                                  P.col_kskb + ((size_t)kvh * P.n_k_tiles + j) * 2 * BN, KSKB_BYTES, bar(RB_K_FULL + sk));
                if (j >= R_VS) ok = wait(RB_V_EMPTY + sv, j / R_VS - 1);
                if (!ok) break;
                mx::mbar_expect_tx(bar(RB_V_FULL + sv), TILE_BYTES);
                mx::tma_load_3d(smem_base + R_SMEM_V + sv * TILE_BYTES, &tmV, bar(RB_V_FULL + sv), 0, j * BN, kvh);
            }
        }
        __syncwarp();
    } else if (warp == SOFT_WARPS + 1) {
        // ------------------------- MMA issuer 1: S = Q K^T --------------
        constexpr uint32_t IDESC_S = mx::mma_idesc_bf16(R_ROWS, BN, false, false);
        const uint64_t a = mx::smem_desc_sw128(smem_base + R_SMEM_Q);
        mx::pdl_wait();
        ok = wait_warp(RB_Q_FULL, 0);
        for (int i = 0, j = 0; j < n && ok; ++i) {
#pragma unroll
            for (int w = 0; w < R_GROUPS; ++w, ++j) {
                if (!ok || j >= n) continue;
                const int s = j % R_KS;
                ok = wait_warp(RB_K_FULL + s, j / R_KS);
                if (ok && i > 0) ok = wait_warp(RB_S_FREE + w, i - 1);
                if (!ok) continue;
                mx::tc_fence_after();
                const uint64_t b = mx::smem_desc_sw128(smem_base + R_SMEM_K + s * TILE_BYTES);
                if (ISSUER_LANE) {
#pragma unroll
                    for (int k = 0; k < HD / 16; ++k) mx::mma_ws_ss(tmem + R_TM_S + w * (BN / 2), a + 2 * k, b + 2 * k, IDESC_S, k > 0);
                    mx::mma_commit(bar(RB_S_FULL + w));
                    mx::mma_commit(bar(RB_K_EMPTY + s));
                }
            }
        }
        __syncwarp();
    } else if (warp == SOFT_WARPS + 2) {
        // ------------------------- MMA issuer 2: O += P V, in key order --
        constexpr uint32_t IDESC_O = mx::mma_idesc_bf16(R_ROWS, HD, false, true);
        mx::pdl_wait();
        const bool own_o = !head_fast();   // each group sums into an O of its own
        for (int i = 0, j = 0; j < n && ok; ++i) {
#pragma unroll
            for (int w = 0; w < R_GROUPS; ++w, ++j) {
                if (!ok || j >= n) continue;
                const int s = j % R_VS;
                ok = wait_warp(RB_V_FULL + s, j / R_VS);
                if (ok) ok = wait_warp(RB_P_FULL + w, i);
                if (!ok) continue;
                mx::tc_fence_after();
                const uint64_t b = mx::smem_desc_sw128(smem_base + R_SMEM_V + s * TILE_BYTES);
                const uint64_t a = mx::smem_desc_sw128(smem_base + R_SMEM_P + w * R_P_BYTES);
                if (ISSUER_LANE) {
#pragma unroll
                    for (int k = 0; k < BN / 16; ++k)   // 16 keys: 32 bytes of P's rows, the second 64 keys in its second tile
                        mx::mma_ws_ss(tmem + R_TM_O + (own_o ? w * (HD / 2) : 0), a + (k >> 2) * (R_P_BYTES / 2 / 16) + 2 * (k & 3),
                                      b + 128 * k, IDESC_O, (own_o ? i > 0 : j > 0) || k > 0);
                    mx::mma_commit(bar(RB_P_DONE + w));
                    mx::mma_commit(bar(RB_V_EMPTY + s));
                }
            }
        }
        __syncwarp();
    } else {
        // ------------------------- softmax groups -----------------------
        const int w = warp >> 2, half = (warp >> 1) & 1, row_in_tile = (warp & 1) * 32 + lane, thr = tid & 127;
        const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
        const uint32_t tm_s = tmem + lane_off + R_TM_S + w * (BN / 2);
        const uint32_t tm_o = tmem + lane_off + R_TM_O;
        const int p_off = R_SMEM_P + w * R_P_BYTES + half * (R_P_BYTES / 2) + row_in_tile * 128;   // this thread's row of P
        const int n_w = (n + R_GROUPS - 1 - w) / R_GROUPS;   // the group's tiles: w, w + 4, ...
        const int row = q0 + row_in_tile;
        const int last = P.causal ? min(N - 1, row + P.q_off) : N - 1;   // last visible key of this row
        uint32_t xmc = 0;            // row-max exchanges of this group so far
        // what group `of` (1..3) handed on with its tile `i`: group 1 and 3 | 2: [sum over the chain before, the tile's sum]; with a
        // row max [sum, max].  A slot is written again four tiles of its group later, when it has been read.
        auto slot = [&](int of, int i, int what) -> float & {
            return ((float *)(smem + R_SMEM_SUM))[(((of - 1) * R_SLOTS + (i & (R_SLOTS - 1))) * 2 + what) * 128 + thr];
        };
        mx::pdl_wait();
        const bool fast = head_fast();
        float row_a = 0.0f, row_qsum = 0.0f;
        if (SRC == SRC_I8 && row < NQ) {
            row_a = P.row_a[(size_t)bh * NQ + row];
            row_qsum = P.row_qsum[(size_t)bh * NQ + row];
        }
        auto kskb_of = [&](int j) {
            return (const float *)(smem + R_SMEM_KSKB + (j % KSKB_SLOTS) * KSKB_BYTES) + half * (BN / 2);
        };
        auto row_max = [&](float own) -> float {   // over the halves of the row
            float *xm = (float *)(smem + R_SMEM_XMAX) + (w * 2 + (xmc & 1)) * 128;
            xm[thr] = own;
            __syncwarp();
            if (lane == 0) mx::mbar_arrive(bar(RB_XMAX + w));
            ok = wait_warp(RB_XMAX + w, xmc);
            ++xmc;
            return fmaxf(own, xm[thr ^ 64]);
        };
        float m = fast ? 0.0f : -CUDART_INF_F, l = 0.0f, corr = 0.0f;
        // The reference of the max-free loop (sources that have one) is the row's max over key tile 0, which the first group
        // publishes.
        float *ref = (float *)(smem + R_SMEM_REF);
        if (REF && SRC != SRC_RAW && fast && w > 0 && n_w > 0) {
            ok = wait_warp(RB_REF, 0);
            if (ok) m = ref[row_in_tile];
        }
        // the group's P buffer is free: P V of its previous tile is complete (usually for long: one cheap look first, 1.5 to 3 % of a
        // long range, 1024 tokens over 30000 fp32 keys 131.1 -> 126.7 us)
        auto p_free = [&](int i) {
            return i == 0 || (bool)__all_sync(0xFFFFFFFFu, mx::mbar_wait_fast(bar(RB_P_DONE + w), (i - 1) & 1, abort_flag, P.status));
        };
        auto put = [&](const uint32_t *pk, int at0) {   // 32 probabilities: four 16-byte pieces of the row, from piece at0 on
#pragma unroll
            for (int i = 0; i < 4; ++i)
                *(uint4 *)(smem + p_off + (((at0 + i) ^ (lane & 7)) << 4)) = make_uint4(pk[4 * i], pk[4 * i + 1], pk[4 * i + 2], pk[4 * i + 3]);
        };
        auto hand_p = [&]() {
            mx::fence_proxy_async_smem();   // read by the MMAs
            __syncwarp();
            if (lane == 0) mx::mbar_arrive(bar(RB_P_FULL + w));
        };
        uint32_t va[32], vb[32];
        float s_prev = 0.0f;   // sum of the group's previous tile, not yet in l
        if (fast) {
            // Sums: l of group 0 (1) is that over even (odd) key tiles in key order.  With its tile i the group takes in
            // tile i - 2 of its partner, group 2 (3), and tile i - 1 of its own: P V of those, and so their sums, precede
            // P V of its tile i - 1, which p_free has waited for.
            float nmc = REF ? -m * c : 0.0f;
            auto sum_of = [](uint64_t v) {
                float a0, a1;
                mx::upk2(v, a0, a1);
                return a0 + a1;
            };
            auto tile = [&](auto first_c, int i) -> bool {
                constexpr bool FIRST = decltype(first_c)::value;   // of the item: key tile 0
                const int j = R_GROUPS * i + w;
                if (!wait_warp(RB_S_FULL + w, i)) return false;
                mx::tc_fence_after();
                mx::tmem_ld32(tm_s, va);
                mx::tmem_wait_ld();
                mx::tmem_ld32(tm_s + 32, vb);   // lands under the first exponentials
                const int key0 = j * BN, col0 = key0 + half * (BN / 2);
                const bool need_mask = (key0 + BN > N) || (P.causal && key0 + BN - 1 > q0 + P.q_off);
                const float *kskb = SRC == SRC_I8 ? kskb_of(j) : nullptr;
                uint64_t rs2;
                uint32_t pk[16];
                constexpr bool LEAD = REF && FIRST;
                if (LEAD) {
                    mx::tmem_wait_ld();
                    if (SRC == SRC_I8) fwd_rebuild32(va, kskb, 0.0f, row_a, row_qsum), fwd_rebuild32(vb, kskb + 32, 0.0f, row_a, row_qsum);
                    if (need_mask) fwd_mask64(va, vb, col0, last);
                    m = row_max(fwd_max64(va, vb));
                    if (!ok) return false;
                    if (half == 0) ref[row_in_tile] = m;
                    __syncwarp();
                    if (lane == 0) mx::mbar_arrive(bar(RB_REF));
                    nmc = -m * c;
                }
                fwd_exp32<SRC>(va, pk, col0, last, need_mask, kskb, true, LEAD, nmc, row_a, row_qsum, rs2);
                mx::tmem_wait_ld();
                mx::tc_fence_before();
                __syncwarp();
                if (lane == 0) mx::mbar_arrive(bar(RB_S_FREE + w));   // this group's columns have left S
                if (!p_free(i)) return false;
                if (w < 2) {
                    if (i >= 2) l += slot(w + 2, i - 2, 1);
                    if (i >= 1) l += s_prev;
                }
                put(pk, 0);
                float rb[4] = {0.0f, 0.0f, 0.0f, 0.0f};   // the first key tile's ROUNDED probabilities (see flash_fwd_kernel)
                auto sum_rounded16 = [&]() {
#pragma unroll
                    for (int u = 0; u < 16; ++u) mx::add_bf16x2(pk[u], rb[(u & 1) * 2], rb[(u & 1) * 2 + 1]);
                };
                if (FIRST) sum_rounded16();
                fwd_exp32<SRC>(vb, pk, col0 + 32, last, need_mask, kskb + 32, false, LEAD, nmc, row_a, row_qsum, rs2);
                put(pk, 4);
                s_prev = sum_of(rs2);
                if (FIRST) {
                    sum_rounded16();
                    corr = ((rb[0] + rb[1]) + (rb[2] + rb[3])) - s_prev;
                }
                if (w > 0) {
                    if (w == 1) slot(1, i, 0) = l;
                    slot(w, i, 1) = s_prev;
                }
                hand_p();
                return true;
            };
            int i = 0;
            if (w == 0) ok = ok && tile(std::true_type{}, i++);
            for (; ok && i < n_w; ++i) ok = tile(std::false_type{}, i);
        } else {
            // ---- running row max, raised lazily: every group has its own, over its key tiles, and its own O ----
            for (int i = 0; ok && i < n_w; ++i) {
                const int j = R_GROUPS * i + w;
                ok = wait_warp(RB_S_FULL + w, i);
                if (!ok) break;
                mx::tc_fence_after();
                mx::tmem_ld32(tm_s, va);
                mx::tmem_ld32(tm_s + 32, vb);
                mx::tmem_wait_ld();
                mx::tc_fence_before();
                __syncwarp();
                if (lane == 0) mx::mbar_arrive(bar(RB_S_FREE + w));
                const int key0 = j * BN, col0 = key0 + half * (BN / 2);
                if (SRC == SRC_I8) {
                    const float *kskb = kskb_of(j);
                    fwd_rebuild32(va, kskb, 0.0f, row_a, row_qsum);
                    fwd_rebuild32(vb, kskb + 32, 0.0f, row_a, row_qsum);
                }
                if ((key0 + BN > N) || (P.causal && key0 + BN - 1 > q0 + P.q_off)) fwd_mask64(va, vb, col0, last);
                const float mx_ = row_max(fwd_max64(va, vb));
                if (!ok) break;
                const bool raise = (i == 0) || ((mx_ - m) * c > RESCALE_LOG2);
                const float m_new = raise ? mx_ : m;
                const float alpha = (raise && i > 0) ? mx::ex2((m - m_new) * c) : 1.0f;
                const float nmc = m_new == -CUDART_INF_F ? 0.0f : -m_new * c;   // (a row may see none of the group's first keys)
                ok = p_free(i);
                if (!ok) break;
                if (i > 0 && __any_sync(0xFFFFFFFFu, raise)) {   // this thread's 32 columns of the group's O
                    mx::tc_fence_after();
#pragma unroll 1
                    for (int cc = 0; cc < 2; ++cc) {
                        uint32_t o[16];
                        mx::tmem_ld16(tm_o + w * (HD / 2) + cc * 16, o);
                        mx::tmem_wait_ld();
#pragma unroll
                        for (int u = 0; u < 16; ++u) o[u] = __float_as_uint(__uint_as_float(o[u]) * alpha);
                        mx::tmem_st16(tm_o + w * (HD / 2) + cc * 16, o);
                    }
                    mx::tmem_wait_st();
                }
                float rs[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                uint32_t pk[16];
                auto exp_general = [&](const uint32_t *v, int piece) {
#pragma unroll
                    for (int u = 0; u < 32; u += 2) {
                        const float p0 = mx::ex2(fmaf(__uint_as_float(v[u]), c, nmc));
                        const float p1 = mx::ex2(fmaf(__uint_as_float(v[u + 1]), c, nmc));
                        rs[u & 2] += p0;
                        rs[(u & 2) + 1] += p1;
                        pk[u >> 1] = mx::pack_bf16(p0, p1);
                    }
                    put(pk, piece);
                };
                exp_general(va, 0);
                exp_general(vb, 4);
                l = l * alpha + ((rs[0] + rs[1]) + (rs[2] + rs[3]));
                m = m_new;
                if (w > 0) slot(w, i, 0) = l, slot(w, i, 1) = m;
                mx::tc_fence_before();
                hand_p();
            }
        }
        // ---- the first group joins the sums and takes O out: thread = row, 32 of its columns ----
        if (ok && w == 0) {
            int n_of[R_GROUPS];
#pragma unroll
            for (int u = 0; u < R_GROUPS; ++u) n_of[u] = (n + R_GROUPS - 1 - u) / R_GROUPS;
            const int e = (n - 1) & (R_GROUPS - 1);   // group of the last key tile
            ok = wait_warp(RB_P_DONE, n_w - 1);       // (first its own last tile: P V of the last group's tile before precedes it)
            if (ok && e > 0) ok = wait_warp(RB_P_DONE + e, (e == 1 ? n_of[1] : e == 2 ? n_of[2] : n_of[3]) - 1);
            mx::tc_fence_after();
            float wt[R_GROUPS] = {1.0f, 0.0f, 0.0f, 0.0f}, l_odd = 0.0f;
            if (ok && fast) {
                if (n_of[0] >= 2) l += slot(2, n_of[0] - 2, 1);
                l += s_prev;
                if (n_of[2] == n_of[0]) l += slot(2, n_of[0] - 1, 1);
                if (n_of[1] > 0) {
                    l_odd = slot(1, n_of[1] - 1, 0);
                    if (n_of[1] >= 2) l_odd += slot(3, n_of[1] - 2, 1);
                    l_odd += slot(1, n_of[1] - 1, 1);
                    if (n_of[3] == n_of[1]) l_odd += slot(3, n_of[1] - 1, 1);
                }
            } else if (ok) {
                float mm = m;
#pragma unroll
                for (int u = 1; u < R_GROUPS; ++u)
                    if (n_of[u] > 0) mm = fmaxf(mm, slot(u, n_of[u] - 1, 1));
                wt[0] = mx::ex2((m - mm) * c);   // m is finite: key tile 0 has a key that every row sees
                l *= wt[0];
#pragma unroll
                for (int u = 1; u < R_GROUPS; ++u)
                    if (n_of[u] > 0) {
                        wt[u] = mx::ex2((slot(u, n_of[u] - 1, 1) - mm) * c);
                        l += slot(u, n_of[u] - 1, 0) * wt[u];
                    }
                m = mm;
            }
            // the halves of a row
            float *xe = (float *)(smem + R_SMEM_END);
            xe[thr] = l, xe[128 + thr] = l_odd, xe[256 + thr] = corr;
            __syncwarp();
            if (lane == 0) mx::mbar_arrive(bar(RB_END));
            if (ok) ok = wait_warp(RB_END, 0);
            if (ok) {
                l = (l + xe[thr ^ 64]) + (l_odd + xe[128 + (thr ^ 64)]);
                const float inv = 1.0f / (l + (corr + xe[256 + (thr ^ 64)]));
                mx::tmem_ld32(tm_o, va);
                mx::tmem_wait_ld();
                if (!fast) {
#pragma unroll
                    for (int i = 0; i < 32; ++i) va[i] = __float_as_uint(__uint_as_float(va[i]) * wt[0]);
#pragma unroll
                    for (int u = 1; u < R_GROUPS; ++u) {
                        if (n_of[u] == 0) continue;
                        mx::tmem_ld32(tm_o + u * (HD / 2), vb);
                        mx::tmem_wait_ld();
#pragma unroll
                        for (int i = 0; i < 32; ++i) va[i] = __float_as_uint(fmaf(__uint_as_float(vb[i]), wt[u], __uint_as_float(va[i])));
                    }
                }
                mx::tc_fence_before();
                float4 o4[8];
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    o4[i] = make_float4(__uint_as_float(va[4 * i]) * inv, __uint_as_float(va[4 * i + 1]) * inv,
                                        __uint_as_float(va[4 * i + 2]) * inv, __uint_as_float(va[4 * i + 3]) * inv);
                if (HALF && row < NQ) {
                    uint4 *dst = (uint4 *)(P.O_half + ((size_t)bh * NQ + row) * HD + half * 32);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const __half2 h2[4] = {__floats2half2_rn(o4[2 * i].x, o4[2 * i].y), __floats2half2_rn(o4[2 * i].z, o4[2 * i].w),
                                               __floats2half2_rn(o4[2 * i + 1].x, o4[2 * i + 1].y), __floats2half2_rn(o4[2 * i + 1].z, o4[2 * i + 1].w)};
                        dst[i] = *(const uint4 *)h2;
                    }
                }
                if (P.tma_out) {
                    // every warp stages its 32 rows and 32 columns in its own rows of the group's P buffer
                    const int wrow0 = q0 + (warp & 1) * 32, st_off = p_off - lane * 128;
#pragma unroll
                    for (int i = 0; i < 8; ++i) *(float4 *)(smem + st_off + lane * 128 + ((i ^ (lane & 7)) << 4)) = o4[i];
                    mx::fence_proxy_async_smem();
                    __syncwarp();
                    if (lane == 0 && wrow0 < NQ) {
                        mx::tma_store_3d(&tmO, smem_base + st_off, half * 32, wrow0, bh);
                        mx::bulk_commit_group();   // (waited for before the kernel ends)
                    }
                } else if (row < NQ) {
                    float *orow = P.O + (size_t)bh * P.o_head_stride + (size_t)row * P.o_row_stride + half * 32;
#pragma unroll
                    for (int i = 0; i < 8; ++i) *(float4 *)(orow + 4 * i) = o4[i];
                }
                if (half == 0 && P.L != nullptr && row < NQ) P.L[(size_t)bh * NQ + row] = m * l_scale + __logf(l);
            }
        }
        if (w == 0 && lane == 0) mx::bulk_wait_group_read<0>();
        __syncwarp();
    }

    // ------------------------- teardown ---------------------------------
    mx::tc_fence_before();
    __syncthreads();
    mx::tc_fence_after();
    mx::pdl_trigger();   // (at the very end, as in flash_fwd_kernel)
    if (warp == SOFT_WARPS + 1) mx::tmem_dealloc(tmem, TM_COLS);
}

// Largest |q|^2 |k|^2 scale^2 log2(e)^2 over the rows of a head of bf16 Q and K -> L[head][every 64th row], the first row
// of an item or query tile in every form, where the forward looks for it (its own scratch would be shared by the streams of a handle; L is the call's).  A
// cluster per head, eight threads per row; bound by the latency of its loads (24 heads of 2048 rows: about 4 us) or, from some
// 20 MB on, by HBM.  A warp stops at the first pass that shows the head beyond the bound (what is left in L is then a part of
// the product, beyond it as well).  Forward of heads beyond the bound, us a call, whole pass / stopping: 1 x 32768 rows
// 554 / 523, 1 x 8192 83 / 77, 24 x 2048 67 / 66, 48 x 4096 causal 229 / 217, 96 x 2048 causal 131 / 127; without any bound pass
// the general loop of an earlier build took 567, 103, 85, 215 and 123.  Heads inside it: 372, 62, 55, 151, 94 (557, 99, 79, 202, 117).
constexpr int RB_THREADS = 256, RB_CLUSTER = 8;
__global__ void __launch_bounds__(RB_THREADS) raw_bounds_kernel(const uint4 *Q, const uint4 *K, float *L, int n) {
    __shared__ int most[2];
    const int tid = threadIdx.x, rank = blockIdx.x, bh = blockIdx.y;
    mx::pdl_trigger();
    if (tid < 2) most[tid] = 0;
    __syncthreads();
    mx::cluster_arrive_release();
    mx::pdl_wait();
    const size_t base = (size_t)bh * n * 8;   // uint4s of 8 values
    const int c = tid & 7;
    int best[2] = {0, 0};   // squared norms as ordered integers (NaN largest)
    auto norm2 = [&](const uint4 &v) {
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
        float ss = 0.0f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float a = __uint_as_float(w[i] << 16), b = __uint_as_float(w[i] & 0xFFFF0000u);
            ss = fmaf(a, a, fmaf(b, b, ss));
        }
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) ss += __shfl_xor_sync(0xFFFFFFFFu, ss, o);   // the row's eight threads
        return __float_as_int(ss) & 0x7FFFFFFF;
    };
    constexpr int STEP = RB_CLUSTER * RB_THREADS / 8, U = 4;   // rows per pass, passes in flight
    for (int r0 = 0; r0 < n; r0 += U * STEP) {
        uint4 q[U], k[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int r = r0 + u * STEP + rank * (RB_THREADS / 8) + (tid >> 3);
            q[u] = k[u] = make_uint4(0, 0, 0, 0);
            if (r < n) q[u] = Q[base + (size_t)r * 8 + c], k[u] = K[base + (size_t)r * 8 + c];
        }
#pragma unroll
        for (int u = 0; u < U; ++u) best[0] = max(best[0], norm2(q[u])), best[1] = max(best[1], norm2(k[u]));
        // beyond the bound already: the rest can only add to it, and the head takes the general loop
        const float seen = __int_as_float(__reduce_max_sync(0xFFFFFFFFu, best[0])) * __int_as_float(__reduce_max_sync(0xFFFFFFFFu, best[1]));
        if (!(seen * (MX230_QK_LOG2_SCALE * MX230_QK_LOG2_SCALE) <= FAST_BOUND_REF * FAST_BOUND_REF)) break;
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        best[i] = __reduce_max_sync(0xFFFFFFFFu, best[i]);
        if ((tid & 31) == 0) atomicMax(&most[i], best[i]);
    }
    __syncthreads();
    mx::cluster_wait();
    if (rank != 0 && tid < 2) mx::cluster_red_max(mx::cluster_map(mx::smem_u32(&most[tid]), 0), most[tid]);
    mx::cluster_sync();
    if (rank != 0) return;
    const float bound = __int_as_float(most[0]) * __int_as_float(most[1]) * (MX230_QK_LOG2_SCALE * MX230_QK_LOG2_SCALE);
    for (int r = tid * (BM / 2); r < n; r += RB_THREADS * (BM / 2)) L[(size_t)bh * n + r] = bound;
}

// fp32 -> bf16 (round to nearest even) for up to four equally sized tensors of `heads` x `per_head4` float4s.
struct CastParams {
    const float *src[4];
    __nv_bfloat16 *dst[4];
    size_t per_head4;   // float4s per head (the whole tensor when heads == 1)
    float4 *zero;       // optional: a buffer of the tensors' size set to zero by one more slice of the grid (blockIdx.y = n_tensors)
    float *norm2[2];    // optional, tensors 0 and 1: [heads][MX230_NORM_PARTS] largest squared row norm seen by each grid part
    int n_tensors;
    float scale0;       // tensor 0 is multiplied by this before rounding (1 = plain cast)
};

// Grid (parts, tensors [+ 1], heads): a block converts every gridDim.x-th group of 256 float4s of its head.  Four
// coalesced 16-byte loads in flight per thread (streaming: the fp32 operands are not needed again and should not push
// the bf16 copies, which the attention kernels read next, out of L2), 8-byte stores.  A row of 64 values is 16
// neighbouring lanes, so its squared norm costs four shuffles on a kernel that waits for memory anyway.
__global__ void __launch_bounds__(256) cast_bf16_kernel(const CastParams P) {
    mx::pdl_trigger();
    mx::pdl_wait();
    const size_t n4 = P.per_head4;
    const size_t base = (size_t)blockIdx.z * n4;
    const size_t step = (size_t)gridDim.x * blockDim.x;
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if ((int)blockIdx.y == P.n_tensors) {
        for (; i < n4; i += step) P.zero[base + i] = make_float4(0.f, 0.f, 0.f, 0.f);
        return;
    }
    const float4 *src = (const float4 *)P.src[blockIdx.y] + base;
    uint2 *dst = (uint2 *)P.dst[blockIdx.y] + base;
    const float sc = blockIdx.y == 0 ? P.scale0 : 1.0f;   // one rounding either way: fp32 product -> bf16
    float *norm_out = blockIdx.y < 2 ? P.norm2[blockIdx.y] : nullptr;
    const unsigned half_mask = 0xFFFFu << (threadIdx.x & 16);   // the 16 lanes that hold one row
    float mx = 0.0f;
    auto row_norm = [&](const float4 &a) {
        float q = a.x * a.x + a.y * a.y + a.z * a.z + a.w * a.w;
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) q += __shfl_xor_sync(half_mask, q, o);
        mx = fmaxf(mx, q);
    };
    for (; i + 3 * step < n4; i += 4 * step) {
        float4 a[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) a[u] = __ldcs(src + i + u * step);
#pragma unroll
        for (int u = 0; u < 4; ++u)
            dst[i + u * step] = make_uint2(mx::pack_bf16(a[u].x * sc, a[u].y * sc), mx::pack_bf16(a[u].z * sc, a[u].w * sc));
        if (norm_out != nullptr) {
#pragma unroll
            for (int u = 0; u < 4; ++u) row_norm(a[u]);
        }
    }
    if (i < n4) {   // the last one to three of a ragged head, their loads together as well
        float4 a[3];
#pragma unroll
        for (int u = 0; u < 3; ++u) a[u] = __ldcs(src + (i + u * step < n4 ? i + u * step : i));
#pragma unroll
        for (int u = 0; u < 3; ++u) {
            if (u > 0 && i + u * step >= n4) break;
            dst[i + u * step] = make_uint2(mx::pack_bf16(a[u].x * sc, a[u].y * sc), mx::pack_bf16(a[u].z * sc, a[u].w * sc));
            if (norm_out != nullptr) row_norm(a[u]);
        }
    }
    if (norm_out != nullptr) {   // block maximum -> this part's slot (parts the grid does not have are set to 0)
        __shared__ float red[8];
        __syncwarp();
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, o));
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int w = 1; w < 8; ++w) mx = fmaxf(mx, red[w]);
            norm_out[(size_t)blockIdx.z * MX230_NORM_PARTS + blockIdx.x] = mx;
            if (blockIdx.x == 0)
                for (int q = (int)gridDim.x; q < MX230_NORM_PARTS; ++q) norm_out[(size_t)blockIdx.z * MX230_NORM_PARTS + q] = 0.0f;
        }
    }
}

}  // namespace

int mx230_launch_cast(mx230_handle *h, cudaStream_t st, const float *const *src, void *const *dst,
                      int n_tensors, int heads, size_t per_head, float *zero, float scale0, float *const *norm2) {
    MX_REQUIRE(per_head % 8 == 0, MX230_ERR_INVALID_ARG, "cast: element count must be a multiple of 8");
    MX_REQUIRE(norm2 == nullptr || per_head % 64 == 0, MX230_ERR_INVALID_ARG, "cast: row norms need rows of 64 values");
    if (per_head == 0 || n_tensors == 0 || heads == 0) return MX230_OK;
    MX_REQUIRE(heads > 0 && heads <= 65535, MX230_ERR_UNSUPPORTED, "cast: %d heads", heads);
    CastParams P;
    for (int i = 0; i < 4; ++i) {
        P.src[i] = src[i < n_tensors ? i : 0];
        P.dst[i] = (__nv_bfloat16 *)dst[i < n_tensors ? i : 0];
        MX_REQUIRE((((uintptr_t)P.src[i] | (uintptr_t)P.dst[i]) & 15) == 0, MX230_ERR_INVALID_ARG,
                   "cast: buffers must be 16-byte aligned");
    }
    P.per_head4 = per_head / 4;
    P.zero = (float4 *)zero;
    P.n_tensors = n_tensors;
    P.scale0 = scale0;
    P.norm2[0] = norm2 ? norm2[0] : nullptr;
    P.norm2[1] = norm2 && n_tensors > 1 ? norm2[1] : nullptr;
    MX_REQUIRE(((uintptr_t)zero & 15) == 0, MX230_ERR_INVALID_ARG, "cast: buffers must be 16-byte aligned");
    // parts per head: every thread gets at least one round of four loads, the whole grid about eight blocks per SM
    const int slices = n_tensors + (zero ? 1 : 0);
    size_t want = (P.per_head4 + 1023) / 1024;
    size_t cap = ((size_t)h->sm_count * 8 + (size_t)slices * heads - 1) / ((size_t)slices * heads);
    size_t parts = want < cap ? want : cap;
    if (parts < 1) parts = 1;
    if (norm2 != nullptr && parts > MX230_NORM_PARTS) parts = MX230_NORM_PARTS;
    if (parts > 65535) parts = 65535;
    MX_LAUNCH(h, st, MX230_K_CAST, mx_launch(cast_bf16_kernel, dim3((unsigned)parts, slices, heads), 256, 0, st, 1, true, P));
    return MX230_OK;
}

namespace {

// Which form a call takes.  Work is counted in 128 x 128 score tiles; the items of a form go to the SMs heaviest first in
// snake order, and the call takes as long as the fullest SM.  A pair item (two query tiles) costs the tiles of both (one and
// a half times the tiles where it has only one: half the softmax groups idle), a key-split item 1.2 times those of its query
// tile (it reads every K/V tile for one query tile only) plus two.  Key-split items are half as large, so they even out
// calls with few items.  Measured (us a call, pair / key-split; 12 heads unless given): 1000 rows causal 18.7 / 15.7, 2048
// rows causal 30.3 / 24.4, 1 x 8192 rows 76 / 51, 4096 rows causal 52.6 / 57.4, 24 x 4096 rows causal 93 / 108, 48 x 4096 rows
// causal 165 / 198.  Over 110 such pairs of timings the rule costs 0.1 % on average, 6 % at most.
bool fwd_key_split(int heads, int n_q, int n_k, int q_off, int causal, int sms) {
    const int tiles = (n_q + BM - 1) / BM, pairs = (tiles + 1) / 2, n_kv = (n_k + BN - 1) / BN;
    if (sms > 256 || (long long)pairs * heads > 4LL * sms) return false;
    auto iters = [&](int t) {
        if (!causal) return n_kv;
        const long long k = ((long long)t * BM + BM - 1 + q_off) / BN + 1;
        return (int)(k < n_kv ? k : n_kv);
    };
    auto fullest = [&](bool split) {
        long long load[256] = {}, most = 0;
        const int blocks = split ? tiles : pairs;
        for (int rank = 0, i = 0; rank < blocks; ++rank) {
            const int b = causal ? blocks - 1 - rank : rank;
            long long cost;   // in tenths of a tile
            if (split) cost = 12LL * iters(b) + 20;
            else cost = 2 * b + 1 < tiles ? 10LL * (iters(2 * b) + iters(2 * b + 1)) : 15LL * iters(2 * b);
            for (int h = 0; h < heads; ++h, ++i) {
                const int r = i / sms, c = (r & 1) ? sms - 1 - i % sms : i % sms;
                load[c] += cost;
                most = load[c] > most ? load[c] : most;
            }
        }
        return most;
    };
    return fullest(true) < fullest(false);
}

// Items of 64 rows wherever every one of them has an SM to itself: a key tile costs such an item less than a key-split item's
// turn of two tiles (980 to 1100 cycles against 2 x 1275), but more per row, so a second round would lose (with a loop over items 12 x 1024 15.2 / 16.6,
// 8 x 2000 21.8 / 24.5, 4 x 4096 30.4 / 30.0).  us a call, key-split / 64 rows.  Heads inside the bound: 1 x 8192 rows causal 48.9 /
// 39.4, 4 x 1024 11.9 / 10.1, 6 x 1400 15.2 / 13.6, 12 x 768 no mask 11.8 / 11.8, prefill of 512 tokens over fp32 keys, 14/2 heads,
// none before them 11.0 / 11.0 (the worst), 512 13.9 / 13.2.  Heads beyond it: 1 x 8192 71.5 / 42.4, 12 x 768 13.5 / 11.9.  bf16
// without a bound: 4 x 1900 19.4 / 12.9, 12 x 768 10.3 / 8.4, 24 x 384 8.0 / 6.9.  Int8 scores, inside the bound and beyond: 512
// over 2048 keys 25.7 / 20.5 and 34.1 / 22.2, 128 over 1128 18.1 / 14.6 and 21.8 / 14.9, 512 alone 15.0 / 12.7 and 16.1 / 12.2, 1
// alone 9.4 / 7.7 and 9.6 / 8.3 (36 sizes below 1280 keys: 0.72 to 0.86 of the key-split form's time, beyond the bound 0.60 to 0.89).
bool fwd_rows64(int heads, int n_q, int sms) { return (long long)((n_q + R_ROWS - 1) / R_ROWS) * heads <= sms; }

template <int SRC, bool KEY_SPLIT, bool HALF = false>
int launch_variant(mx230_handle *h, cudaStream_t st, dim3 grid, const CUtensorMap &tq, const CUtensorMap &tk,
                   const CUtensorMap &tv, const CUtensorMap &to, const FwdParams &P) {
    if constexpr (!HALF && (SRC == SRC_PRE || SRC == SRC_I8))   // (what prefill stages)
        if (P.O_half) return launch_variant<SRC, KEY_SPLIT, true>(h, st, grid, tq, tk, tv, to, P);
    MX_SMEM_ATTR_ONCE(h->device, (flash_fwd_kernel<SRC, KEY_SPLIT, HALF>), SMEM_ALLOC);
    MX_LAUNCH(h, st, MX230_K_FLASH_FWD,
              mx_launch(flash_fwd_kernel<SRC, KEY_SPLIT, HALF>, grid, FWD_THREADS, SMEM_ALLOC, st, 1, true, tq, tk, tv, to, P));
    return MX230_OK;
}

template <int SRC, bool HALF = false>
int launch_rows64(mx230_handle *h, cudaStream_t st, dim3 grid, const CUtensorMap &tq, const CUtensorMap &tk, const CUtensorMap &tv,
                  const CUtensorMap &to, const FwdParams &P) {
    if constexpr (!HALF && (SRC == SRC_PRE || SRC == SRC_I8))
        if (P.O_half) return launch_rows64<SRC, true>(h, st, grid, tq, tk, tv, to, P);
    MX_SMEM_ATTR_ONCE(h->device, (flash_fwd_rows64_kernel<SRC, HALF>), R_ALLOC);
    MX_LAUNCH(h, st, MX230_K_FLASH_FWD,
              mx_launch(flash_fwd_rows64_kernel<SRC, HALF>, grid, FWD_THREADS, R_ALLOC, st, 1, true, tq, tk, tv, to, P));
    return MX230_OK;
}

}  // namespace

// General launcher.  Q: bf16 [heads][n_q][64]; K, V: bf16 [heads / kv_group][n_k][64].
int mx230_launch_flash_fwd_ex(mx230_handle *h, cudaStream_t st, const void *Qb, const void *Kb,
                              const void *Vb, float *O, float *L, int heads, int n_q, int n_k, int q_off,
                              int kv_group, long long o_head_stride, long long o_row_stride, int causal,
                              int q_prescaled, const float *q_norm2, const float *k_norm2, const float *row_a,
                              const float *row_qsum, const float *col_kskb, void *O_half) {
    CUtensorMap tq, tk, tv, to;
    uint64_t rs = HD * 2;
    int rc;
    const bool tma_out = (((uintptr_t)O & 15) == 0) && o_row_stride % 4 == 0 && o_head_stride % 4 == 0 &&
                         o_row_stride > 0 && o_head_stride > 0;
    if (tma_out) {
        if ((rc = mx230_make_tmap_f32_half_rows_strided(h, &to, O, n_q, heads, (uint64_t)o_row_stride * 4,
                                                        (uint64_t)o_head_stride * 4)))
            return rc;
    } else {
        memset(&to, 0, sizeof(to));
    }
    const bool rows64 = fwd_rows64(heads, n_q, h->sm_count);
    const bool key_split = !rows64 && fwd_key_split(heads, n_q, n_k, q_off, causal, h->sm_count);
    if ((rc = mx230_make_tmap_bf16(h, &tq, Qb, n_q, heads, rs, (uint64_t)n_q * HD * 2, rows64 ? R_ROWS : BM))) return rc;
    if ((rc = mx230_make_tmap_bf16(h, &tk, Kb, n_k, heads / kv_group, rs, (uint64_t)n_k * HD * 2, BN))) return rc;
    if ((rc = mx230_make_tmap_bf16(h, &tv, Vb, n_k, heads / kv_group, rs, (uint64_t)n_k * HD * 2, BN))) return rc;
    FwdParams P;
    P.O = O;
    P.O_half = (__half *)O_half;
    P.L = L;
    P.o_head_stride = o_head_stride;
    P.o_row_stride = o_row_stride;
    P.n_q = n_q;
    P.n_k = n_k;
    P.q_off = q_off;
    P.kv_group = kv_group;
    P.causal = causal ? 1 : 0;
    P.heads = heads;
    P.item_rows = rows64 ? R_ROWS : key_split ? BM : QT * BM;
    P.n_qblocks = (n_q + P.item_rows - 1) / P.item_rows;
    MX_REQUIRE((long long)heads * P.n_qblocks <= 0x7FFFFFFF, MX230_ERR_UNSUPPORTED, "flash forward: too many query blocks");
    P.n_items = heads * P.n_qblocks;
    P.tma_out = tma_out ? 1 : 0;
    P.q_norm2 = (q_norm2 && k_norm2) ? q_norm2 : nullptr;
    P.k_norm2 = P.q_norm2 ? k_norm2 : nullptr;
    P.test_drop_tile = h->test_drop_tile;
    // Operands the caller staged come without norms; with L at hand a pass over Q and K bounds the scores.  It is worth its
    // launch from 16 key tiles per row on (a head's row count decides, not the number of heads: a head's bits do not
    // depend on the heads beside it).
    const bool raw_bounds = !row_a && !q_prescaled && L != nullptr && kv_group == 1 && n_q == n_k && n_k > 15 * BN;
    if (raw_bounds)
        MX_LAUNCH(h, st, MX230_K_CAST, mx_launch(raw_bounds_kernel, dim3(RB_CLUSTER, heads), RB_THREADS, 0, st, RB_CLUSTER, true,
                                                 (const uint4 *)Qb, (const uint4 *)Kb, L, n_q));
    P.row_a = row_a;
    P.row_qsum = row_qsum;
    P.col_kskb = col_kskb;
    P.n_k_tiles = (n_k + BN - 1) / BN;
    P.status = h->status_dev;
    // persistent: one CTA per SM (the kernel holds all of an SM's tensor memory), each walking its share of the items; 64-row items
    // have a CTA each
    dim3 grid((unsigned)(rows64 || P.n_items < h->sm_count ? P.n_items : h->sm_count));
    if (rows64) {
        if (row_a) return launch_rows64<SRC_I8>(h, st, grid, tq, tk, tv, to, P);
        if (q_prescaled) return launch_rows64<SRC_PRE>(h, st, grid, tq, tk, tv, to, P);
        return raw_bounds ? launch_rows64<SRC_RAW_BOUND>(h, st, grid, tq, tk, tv, to, P) : launch_rows64<SRC_RAW>(h, st, grid, tq, tk, tv, to, P);
    }
    if (row_a) return key_split ? launch_variant<SRC_I8, true>(h, st, grid, tq, tk, tv, to, P)
                                : launch_variant<SRC_I8, false>(h, st, grid, tq, tk, tv, to, P);
    if (q_prescaled) return key_split ? launch_variant<SRC_PRE, true>(h, st, grid, tq, tk, tv, to, P)
                                      : launch_variant<SRC_PRE, false>(h, st, grid, tq, tk, tv, to, P);
    if (raw_bounds) return key_split ? launch_variant<SRC_RAW_BOUND, true>(h, st, grid, tq, tk, tv, to, P)
                                     : launch_variant<SRC_RAW_BOUND, false>(h, st, grid, tq, tk, tv, to, P);
    return key_split ? launch_variant<SRC_RAW, true>(h, st, grid, tq, tk, tv, to, P)
                     : launch_variant<SRC_RAW, false>(h, st, grid, tq, tk, tv, to, P);
}

int mx230_launch_flash_fwd(mx230_handle *h, cudaStream_t st, const void *Qb, const void *Kb,
                           const void *Vb, float *O, float *L, int batch_heads, int n, int causal,
                           int q_prescaled, const float *q_norm2, const float *k_norm2) {
    return mx230_launch_flash_fwd_ex(h, st, Qb, Kb, Vb, O, L, batch_heads, n, n, 0, 1, (long long)n * HD, HD,
                                     causal, q_prescaled, q_norm2, k_norm2, nullptr, nullptr, nullptr, nullptr);
}

static int check_flash_args(const char *who, mx230_handle *h, int batch_heads, int n) {
    MX_REQUIRE(h != nullptr, MX230_ERR_INVALID_ARG, "%s: null handle", who);
    MX_REQUIRE(batch_heads >= 0 && n >= 0, MX230_ERR_INVALID_ARG, "%s: negative size", who);
    MX_REQUIRE(batch_heads <= 65535, MX230_ERR_UNSUPPORTED, "%s: batch_heads %d > 65535", who,
               batch_heads);
    return MX230_OK;
}

extern "C" int mx230_cast_bf16(mx230_handle *h, void *stream, const float *src, void *dst_bf16,
                               size_t count) {
    MX_REQUIRE(h && (count == 0 || (src && dst_bf16)), MX230_ERR_INVALID_ARG, "cast_bf16: null argument");
    mx230_device_guard guard(h->device);
    const float *s[1] = {src};
    void *d[1] = {dst_bf16};
    return mx230_launch_cast(h, (cudaStream_t)stream, s, d, 1, 1, count, nullptr, 1.0f, nullptr);
}

extern "C" int mx230_attn_flash_bf16(mx230_handle *h, void *stream, const void *Qb, const void *Kb,
                                     const void *Vb, float *O, float *L_or_null, int batch_heads,
                                     int n, int causal) {
    int rc = check_flash_args("attn_flash_bf16", h, batch_heads, n);
    if (rc) return rc;
    if (batch_heads == 0 || n == 0) return MX230_OK;
    MX_REQUIRE(Qb && Kb && Vb && O, MX230_ERR_INVALID_ARG, "attn_flash_bf16: null tensor");
    MX_REQUIRE((((uintptr_t)O) & 15) == 0, MX230_ERR_INVALID_ARG, "attn_flash_bf16: O must be 16-byte aligned");
    mx230_device_guard guard(h->device);
    return mx230_launch_flash_fwd(h, (cudaStream_t)stream, Qb, Kb, Vb, O, L_or_null, batch_heads, n,
                                  causal, 0, nullptr, nullptr);
}

static int flash_fp32(mx230_handle *h, void *stream, const float *Q, const float *K, const float *V,
                      float *O, float *L, int batch_heads, int n, int causal, const char *who) {
    int rc = check_flash_args(who, h, batch_heads, n);
    if (rc) return rc;
    if (batch_heads == 0 || n == 0) return MX230_OK;
    MX_REQUIRE(Q && K && V && O, MX230_ERR_INVALID_ARG, "%s: null tensor", who);
    size_t need = mx230_flash_workspace_bytes(batch_heads, n, 0);
    MX_REQUIRE(h->ws && need <= h->ws_bytes, MX230_ERR_WORKSPACE,
               "%s: workspace %zu B < %zu B needed (call mx230_reserve)", who, h->ws_bytes, need);
    mx230_device_guard guard(h->device);
    const size_t one = mx230_flash_stage_bytes(batch_heads, n);
    void *qb = h->ws, *kb = (char *)h->ws + one, *vb = (char *)h->ws + 2 * one;
    float *qn = (float *)((char *)h->ws + 3 * one), *kn = qn + (size_t)batch_heads * MX230_NORM_PARTS;
    const float *src[3] = {Q, K, V};
    void *dst[3] = {qb, kb, vb};
    float *norms[2] = {qn, kn};
    // Q is staged as Q * (scale * log2 e), rounded once from the fp32 product: the kernel's scores are then
    // already in log2 units.  The same launch leaves the largest row norms of Q and K per head, from which the
    // kernel bounds |q . k| and, where the bound allows, runs its softmax loop without a row max.
    h->staged.valid = 0;
    rc = mx230_launch_cast(h, (cudaStream_t)stream, src, dst, 3, batch_heads, (size_t)n * HD, nullptr,
                           MX230_QK_LOG2_SCALE, norms);
    if (rc) return rc;
    h->staged = {Q, K, V, batch_heads, n, 1, nullptr};
    return mx230_launch_flash_fwd(h, (cudaStream_t)stream, qb, kb, vb, O, L, batch_heads, n, causal, 1, qn, kn);
}

extern "C" int mx230_attn_flash(mx230_handle *h, void *stream, const float *Q, const float *K,
                                const float *V, float *O, int batch_heads, int n, int causal) {
    return flash_fp32(h, stream, Q, K, V, O, nullptr, batch_heads, n, causal, "attn_flash");
}

extern "C" int mx230_attn_flash_lse(mx230_handle *h, void *stream, const float *Q, const float *K,
                                    const float *V, float *O, float *L, int batch_heads, int n,
                                    int causal) {
    MX_REQUIRE(L != nullptr || batch_heads == 0 || n == 0, MX230_ERR_INVALID_ARG,
               "attn_flash_lse: null L");
    return flash_fp32(h, stream, Q, K, V, O, L, batch_heads, n, causal, "attn_flash_lse");
}

