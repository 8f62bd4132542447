// The projections either side of the attention step, for one decode token:
//   gemv:            y[o] (+)= sum_i x[i] w[i*n_out + o] + b[o]     (gemv / gemv_half, the output
//                    projection with its fused residual add, 03-llm-engine/kernels/llm.cu:144-177,
//                    host gemv() src/gpu.rs:1158-1198, call site :2676-2686)
//   qkv step, fused: qkv = x W + b, RoPE on the Q and K heads, K and V rows written to the cache
//                    (fp32 copy or int8 quantize-on-write), the rotated q left in qkv for the decode
//                    attention -- one launch for the reference's gemv + rope + KV write
//                    (gpu.rs:2558-2646; rope llm.cu:1072-1100, quant_affine :1137-1149).
//
//   gemv_int8:       the same with int8 weights and on-the-fly int8 activations (llm.cu:226-316): the
//                    activation row is quantised per group of AG values (absmax / 127, round to nearest
//                    even), weights are int32 words of four consecutive input rows, w32[(i/4)*n_out + o],
//                    integer dots by dp4a, one float multiply-add per group, one scale per output column.
//
// The floor is HBM on the weight matrix (n_in x n_out fp32, fp16 or int8, each byte read once); at a decode token's
// sizes (2 MB) the time is latency instead: launch, one memory round trip, the merge of the partial sums.  The reference
// gives one thread a whole output column.  Here a 64-column block (one attention head) is summed in slices of the input
// rows, eight row lanes per slice, lanes and slices added in a fixed order that depends on the sizes alone (a rotated q is
// quantised to int8 downstream, where another last bit can move a code).  Up to 64 slices belong to one thread-block
// cluster of up to eight CTAs, which push their slices' sums into the first one's shared memory, where the epilogue runs;
// more slices go through the workspace, merged by the last CTA to arrive.  The kernel is launched programmatically: its
// slices of the weights are on their way into L2 while the kernel before it still runs.
#include <cuda_fp16.h>

#include "common.cuh"

namespace {

constexpr int PJ_COLS = 64;       // columns per CTA = one head
constexpr int PJ_ROWLANES = 8;    // row lanes of a slice: lane l sums rows l, l + 8, ...
constexpr int PJ_CLUSTER = 8;     // most CTAs of a column block that merge through shared memory
constexpr int PJ_SLOTS = 8;       // most slices of a CTA
constexpr int PJ_SLICES_PER_SM = 6;   // slices, over all column blocks, that the split aims at

struct QkvEpilogue {
    int enabled;
    int pos;                 // host position, unless pos_dev
    const int *pos_dev;
    int n_head, n_kv_head;
    float theta;
    float *kcache, *vcache;  // fp32 cache, or null
    int8_t *kq, *vq;         // int8 cache, or null
    float *ks, *vs, *kb, *vb;
    const int *bt;           // block table or null
    int bs;
};

struct GemvParams {
    float *y;
    const float *x;
    const void *w;
    const float *b;
    int n_in, n_out, accum;
    const float *scales;     // int8 weights: one scale per output column
    int ag;                  // int8 weights: activations are quantised in groups of `ag` values (4 or 8)
    int rows_per_slice, n_slices;   // per column block
    int slots, ctas, cl_size;       // slices per CTA, CTAs per column block; cl_size = ctas, or 1: merge through the workspace
    float *partials;                // [n_slices][n_out]
    unsigned *counters;      // one per column block, self-resetting
    int *status;             // where a wait within a cluster that ran out is recorded
    int test_drop;           // test hook: >= 0: the first column block waits for sums that nobody sends
    QkvEpilogue e;
};

// CPT consecutive columns of one weight row: fp32 (4), fp16 (8, or 4 where rows are only 8-byte aligned) or packed int8
// words (4)
template <typename WT, int CPT>
struct WeightRow;
template <>
struct WeightRow<float, 4> {
    float4 r;
    __device__ __forceinline__ void load(const void *w, size_t i) { r = *(const float4 *)((const float *)w + i); }
    __device__ __forceinline__ void zero() { r = make_float4(0.f, 0.f, 0.f, 0.f); }
    __device__ __forceinline__ void fma(float x, float (&a)[4]) const {
        a[0] = fmaf(x, r.x, a[0]), a[1] = fmaf(x, r.y, a[1]), a[2] = fmaf(x, r.z, a[2]), a[3] = fmaf(x, r.w, a[3]);
    }
};
__device__ __forceinline__ void fma_half2(float x, uint32_t raw, float &a, float &b) {
    const float2 w = __half22float2(*(const __half2 *)&raw);
    a = fmaf(x, w.x, a), b = fmaf(x, w.y, b);
}
template <>
struct WeightRow<__half, 8> {
    uint4 r;
    __device__ __forceinline__ void load(const void *w, size_t i) { r = *(const uint4 *)((const __half *)w + i); }
    __device__ __forceinline__ void zero() { r = make_uint4(0, 0, 0, 0); }
    __device__ __forceinline__ void fma(float x, float (&a)[8]) const {
        fma_half2(x, r.x, a[0], a[1]), fma_half2(x, r.y, a[2], a[3]), fma_half2(x, r.z, a[4], a[5]), fma_half2(x, r.w, a[6], a[7]);
    }
};
template <>
struct WeightRow<__half, 4> {
    uint2 r;
    __device__ __forceinline__ void load(const void *w, size_t i) { r = *(const uint2 *)((const __half *)w + i); }
    __device__ __forceinline__ void zero() { r = make_uint2(0, 0); }
    __device__ __forceinline__ void fma(float x, float (&a)[4]) const {
        fma_half2(x, r.x, a[0], a[1]), fma_half2(x, r.y, a[2], a[3]);
    }
};
template <>
struct WeightRow<int8_t, 4> {
    int4 r;
    __device__ __forceinline__ void load(const void *w, size_t i) { r = *(const int4 *)((const int *)w + i); }
    __device__ __forceinline__ void zero() { r = make_int4(0, 0, 0, 0); }
    __device__ __forceinline__ void fma(int xq, float sx, float (&a)[4]) const {
        a[0] = fmaf((float)__dp4a(r.x, xq, 0), sx, a[0]), a[1] = fmaf((float)__dp4a(r.y, xq, 0), sx, a[1]);
        a[2] = fmaf((float)__dp4a(r.z, xq, 0), sx, a[2]), a[3] = fmaf((float)__dp4a(r.w, xq, 0), sx, a[3]);
    }
};

// Grid: column blocks x CTAs, the CTAs of a block next to each other.  A slice takes 64 / CPT * 8 threads.
// Registers: two CTAs of five slices (640 threads at four columns a thread, 320 at eight) have to fit an SM, so that the next
// launch's are there, with their weights on the way into L2, while this one's still run: 896 -> 1152 fp32, launch after launch
// over fresh weights, 4.6 us at 50 registers (one CTA), 3.2 at 48.  fp16 rows of a multiple of 4 columns take six slices a CTA in
// grids of more CTAs than SMs: two such CTAs of 768 threads at 40 registers (2048 -> 1220, launch after launch: 32 registers 4.0 us,
// 48 5.6, 40 3.9).  int8 keeps its unpacked words in registers (1504 -> 1412: 58 registers 3.2, 48 3.6, 64 3.0; 896 -> 896 3.2, 3.2,
// 3.0).
template <typename WT, int CPT>
__global__ void __maxnreg__(CPT == 8 ? 56 : sizeof(WT) == 2 ? 40 : sizeof(WT) == 1 ? 64 : 48)
gemv_heads_kernel(const GemvParams P) {
    constexpr bool I8 = sizeof(WT) == 1;
    constexpr int TPR = PJ_COLS / CPT;              // threads across a weight row
    constexpr int TPS = TPR * PJ_ROWLANES;          // threads of a slice
    constexpr int BATCH = 4;                        // passes whose loads are issued together
    constexpr int ELT = I8 ? 4 : (int)sizeof(WT);   // bytes of a stored weight word
    constexpr int IN_PER_ROW = I8 ? 4 : 1;          // input rows in one stored row
    __shared__ __align__(16) float red[PJ_SLOTS][PJ_ROWLANES][PJ_COLS];
    __shared__ __align__(16) float parts[PJ_CLUSTER * PJ_SLOTS][PJ_COLS];   // first CTA of the cluster: the sums of every slice
    __shared__ __align__(8) unsigned long long parts_bar;                   // completed by their bytes
    __shared__ int is_last, aborted;
    extern __shared__ float xs[];                   // int8: the CTA's part of x as packed codes, then group scales
    const int tid = threadIdx.x, nt = blockDim.x, C = P.cl_size;
    const int blk = blockIdx.x / P.ctas, rank = blockIdx.x - blk * P.ctas;
    const int col0 = blk * PJ_COLS;
    const int slot = tid / TPS, tl = tid - slot * TPS;
    const int slice = rank * P.slots + slot;
    // input rows of the CTA and of this thread's slice
    const int c0 = min(P.n_in, rank * P.slots * P.rows_per_slice), c1 = min(P.n_in, c0 + P.slots * P.rows_per_slice);
    const int r0 = min(P.n_in, slice * P.rows_per_slice) / IN_PER_ROW;
    const int r1 = min(P.n_in, (slice + 1) * P.rows_per_slice) / IN_PER_ROW;

    mx::pdl_trigger();
    const uint32_t bar = mx::smem_u32(&parts_bar);
    if (C > 1) {
        if (tid == 0) {
            aborted = 0;
            mx::mbar_init(bar, 1);
            mx::mbar_fence_init();
            if (rank == 0) mx::mbar_expect_tx(bar, P.n_slices * PJ_COLS * 4 + (P.test_drop >= 0 && blk == 0 ? 16 : 0));
        }
        mx::cluster_arrive_relaxed();               // waited for before the first store to another CTA's memory
    }
    // start of the CTA's rows into L2 under the previous kernel's tail
    for (int r = c0 / IN_PER_ROW + tid, n = 0; r < c1 / IN_PER_ROW && n < 2; r += nt, ++n) {
        const char *line = (const char *)P.w + ((size_t)r * P.n_out + col0) * ELT;
        mx::prefetch_l2(line);
        if (ELT == 4 && col0 + 32 < P.n_out) mx::prefetch_l2(line + 128);
    }
    const QkvEpilogue &E = P.e;
    const bool finishes = (rank == 0 || C == 1) && tid < 32;   // the warp that finishes the block: lane l has columns 2l and 2l + 1
    const float freq = finishes && E.enabled ? mx::rope_freq(tid, 64, E.theta) : 0.0f;
    mx::pdl_wait();

    const int cq = tl % TPR, rl = tl / TPR;
    const int col = col0 + CPT * cq;
    const bool live = col < P.n_out;                // n_out is a multiple of CPT
    float acc[CPT];
#pragma unroll
    for (int c = 0; c < CPT; ++c) acc[c] = 0.0f;
    WeightRow<WT, CPT> w[BATCH];
    float xv[BATCH];
    auto load = [&](int r) {
#pragma unroll
        for (int u = 0; u < BATCH; ++u) {
            const int i = r + u * PJ_ROWLANES;
            const bool in = live && i < r1;
            if (in) w[u].load(P.w, (size_t)i * P.n_out + col);
            else w[u].zero();
            if (!I8) xv[u] = in ? P.x[i] : 0.0f;
        }
    };
    load(r0 + rl);
    // what the epilogue needs, under the weight loads
    const bool is_v = blk >= E.n_head + E.n_kv_head;
    float bias[2] = {0.0f, 0.0f}, scale_o[2] = {1.0f, 1.0f}, y_old[2] = {0.0f, 0.0f};
    int pos = 0;
    size_t row = 0;
    if (finishes) {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int o = col0 + 2 * tid + k;   // (n_out % 4 == 0)
            if (o >= P.n_out) break;
            if (P.b) bias[k] = P.b[o];
            if (I8) scale_o[k] = P.scales[o];
            if (P.accum) y_old[k] = P.y[o];
        }
        if (E.enabled) {
            pos = E.pos_dev ? *E.pos_dev : E.pos;
            row = E.bt && blk >= E.n_head ? (size_t)(E.bt[pos / E.bs] * E.bs + pos % E.bs) : (size_t)pos;
        }
    }
    if constexpr (I8) {
        // quantise the CTA's part of the activations exactly as the reference kernel does
        const int ag = P.ag;
        int *xq = (int *)xs;                                  // (c1 - c0) / 4 words
        float *xsc = xs + P.slots * P.rows_per_slice / 4;     // (c1 - c0) / ag scales
        for (int g = tid; g < (c1 - c0) / ag; g += nt) {
            const float *xg = P.x + c0 + g * ag;
            float amax = 0.0f;
            for (int j = 0; j < ag; ++j) amax = fmaxf(amax, fabsf(xg[j]));
            const float id = amax > 0.0f ? __fdiv_rn(127.0f, amax) : 0.0f;
            for (int q = 0; q < ag / 4; ++q) {
                int packed = 0;
                for (int j = 0; j < 4; ++j) {
                    const int v = max(-127, min(127, __float2int_rn(xg[4 * q + j] * id)));
                    packed |= (v & 0xFF) << (8 * j);
                }
                xq[g * (ag / 4) + q] = packed;
            }
            xsc[g] = amax > 0.0f ? __fdiv_rn(amax, 127.0f) : 1.0f;
        }
        __syncthreads();
        const int wpg = ag / 4;   // word q holds input rows 4q .. 4q+3; its group scale is xsc[q / wpg]
        for (int r = r0 + rl; r < r1; r += BATCH * PJ_ROWLANES) {
            if (r != r0 + rl) load(r);
#pragma unroll
            for (int u = 0; u < BATCH; ++u) {
                const int q = r + u * PJ_ROWLANES;
                if (q < r1) w[u].fma(xq[q - c0 / 4], xsc[(q - c0 / 4) / wpg], acc);
            }
        }
    } else {
        for (int r = r0 + rl; r < r1; r += BATCH * PJ_ROWLANES) {
            if (r != r0 + rl) load(r);
#pragma unroll
            for (int u = 0; u < BATCH; ++u)
                if (r + u * PJ_ROWLANES < r1) w[u].fma(xv[u], acc);
        }
    }
#pragma unroll
    for (int c = 0; c < CPT; c += 4) *(float4 *)&red[slot][rl][CPT * cq + c] = make_float4(acc[c], acc[c + 1], acc[c + 2], acc[c + 3]);
    __syncthreads();
    // ---- lanes -> slices -> block, each in index order ----
    if (C > 1) mx::cluster_wait();   // every CTA of the cluster runs and has its barrier set up
    for (int i = tid; i < P.slots * (PJ_COLS / 4); i += nt) {
        const int sl = i / (PJ_COLS / 4), c = (i - sl * (PJ_COLS / 4)) * 4, g = rank * P.slots + sl;
        if (g >= P.n_slices) break;
        float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int r = 0; r < PJ_ROWLANES; ++r) {
            const float4 v = *(const float4 *)&red[sl][r][c];
            sum.x += v.x, sum.y += v.y, sum.z += v.z, sum.w += v.w;
        }
        // (asynchronous stores that complete the first CTA's barrier: the cluster barrier behind plain ones took 1500 cycles of
        // the 5000 of a launch)
        if (C > 1) mx::cluster_st_async(mx::cluster_map(mx::smem_u32(&parts[g][c]), 0), mx::cluster_map(bar, 0), sum.x, sum.y, sum.z, sum.w);
        else if (P.ctas == 1) *(float4 *)&parts[g][c] = sum;
        else if (col0 + c < P.n_out) *(float4 *)(P.partials + (size_t)g * P.n_out + col0 + c) = sum;   // (n_out % 4 == 0)
    }
    if (C > 1) {
        if (!finishes) return;   // (see cluster_sums_wait)
    } else if (P.ctas > 1) {
        __threadfence();
        __syncthreads();
        if (tid == 0) is_last = atomicInc(&P.counters[blk], P.ctas - 1) == (unsigned)(P.ctas - 1);
        __syncthreads();
        if (!is_last || !finishes) return;
        __threadfence();
    } else {
        __syncthreads();
        if (!finishes) return;
    }
    // ---- epilogue on the 64 finished sums of this column block: one warp ----
    float cs = 1.0f, sn = 0.0f;
    if (E.enabled && !is_v) mx::rope_angle(pos, freq, cs, sn);   // (while the other CTAs' sums are on their way)
    if (C > 1 && !mx::cluster_sums_wait<false>(bar, &aborted, P.status)) return;   // (nothing is written)
    // (a loop that is short in code as well: what runs once per launch is fetched once per launch)
    const bool in = col0 + 2 * tid < P.n_out;
    float2 sum = make_float2(0.f, 0.f);
    if (P.n_slices == 1) {
        sum = *(const float2 *)&parts[0][2 * tid];
    } else if (C == 1 && P.ctas > 1) {
        if (in)
            for (int g = 0; g < P.n_slices; ++g) {
                const float2 p = __ldcg((const float2 *)(P.partials + (size_t)g * P.n_out + col0 + 2 * tid));
                sum.x += p.x, sum.y += p.y;
            }
    } else {
#pragma unroll 8
        for (int g = 0; g < P.n_slices; ++g) {
            const float2 p = *(const float2 *)&parts[g][2 * tid];
            sum.x += p.x, sum.y += p.y;
        }
    }
    float2 v = make_float2((I8 ? sum.x * scale_o[0] : sum.x) + bias[0], (I8 ? sum.y * scale_o[1] : sum.y) + bias[1]);
    if (!E.enabled) {
        if (P.accum) v.x = y_old[0] + v.x, v.y = y_old[1] + v.y;
        if (in) *(float2 *)(P.y + col0 + 2 * tid) = v;
        return;
    }
    // qkv step: this block is head `blk` of the row [Q heads | K heads | V heads]; lane l owns the rotation pair (l, l + 32)
    float x1, x2;
    {
        const float e1 = __shfl_sync(0xFFFFFFFFu, v.x, tid >> 1), o1 = __shfl_sync(0xFFFFFFFFu, v.y, tid >> 1);
        const float e2 = __shfl_sync(0xFFFFFFFFu, v.x, 16 + (tid >> 1)), o2 = __shfl_sync(0xFFFFFFFFu, v.y, 16 + (tid >> 1));
        x1 = (tid & 1) ? o1 : e1, x2 = (tid & 1) ? o2 : e2;
    }
    if (!is_v) mx::rope_pair(x1, x2, cs, sn);
    P.y[(size_t)blk * 64 + tid] = x1, P.y[(size_t)blk * 64 + 32 + tid] = x2;
    if (blk < E.n_head) return;
    // K or V head: the cache row of this position
    const int kvh = is_v ? blk - E.n_head - E.n_kv_head : blk - E.n_head;
    const int kvd = E.n_kv_head * 64;
    if (E.kq == nullptr) {
        float *dst = (is_v ? E.vcache : E.kcache) + row * kvd + kvh * 64;
        dst[tid] = x1, dst[tid + 32] = x2;
    } else {
        int8_t *dst = (is_v ? E.vq : E.kq) + row * kvd + kvh * 64;
        float *sc = is_v ? E.vs : E.ks, *be = is_v ? E.vb : E.kb;
        const size_t sd = row * E.n_kv_head + kvh;
        int c0, c1;
        float scale, beta;
        mx::quant_head_row(x1, x2, be != nullptr, c0, c1, scale, beta);
        if (tid == 0) {
            sc[sd] = scale;
            if (be != nullptr) be[sd] = beta;
        }
        dst[tid] = (int8_t)c0, dst[tid + 32] = (int8_t)c1;
    }
}

// w_kind: 0 fp32, 1 fp16, 2 int8 (packed words, P.scales and P.ag set)
int launch_gemv(mx230_handle *h, void *stream, GemvParams P, int w_kind, const char *who) {
    MX_REQUIRE(h && P.y && P.x && P.w, MX230_ERR_INVALID_ARG, "%s: null argument", who);
    MX_REQUIRE(P.n_in > 0 && P.n_out > 0 && P.n_out % 4 == 0, MX230_ERR_INVALID_ARG,
               "%s: n_in %d, n_out %d (n_out must be a positive multiple of 4)", who, P.n_in, P.n_out);
    MX_REQUIRE((((uintptr_t)P.w | (uintptr_t)P.y) & 15) == 0, MX230_ERR_INVALID_ARG, "%s: y and w must be 16-byte aligned", who);
    if (w_kind == 2) {
        MX_REQUIRE(P.scales && (P.ag == 4 || P.ag == 8) && P.n_in % 8 == 0, MX230_ERR_INVALID_ARG,
                   "%s: int8 weights need scales, an activation group of 4 or 8 and n_in %% 8 == 0 (n_in %d)", who, P.n_in);
    }
    const int n_blocks = (P.n_out + PJ_COLS - 1) / PJ_COLS;
    // Slices: PJ_SLICES_PER_SM of them per SM over all blocks, at least 16 rows each (int8: whole activation groups and whole
    // passes of the eight row lanes over 4-row words).  This fixes the order of the sums.
    int n_slices = (PJ_SLICES_PER_SM * h->sm_count + n_blocks - 1) / n_blocks;
    const int max_slices = (P.n_in + 15) / 16;
    if (n_slices > max_slices) n_slices = max_slices;
    const int gran = w_kind == 2 ? 4 * PJ_ROWLANES : PJ_ROWLANES;
    P.rows_per_slice = ((P.n_in + n_slices - 1) / n_slices + gran - 1) / gran * gran;
    P.n_slices = n_slices = (P.n_in + P.rows_per_slice - 1) / P.rows_per_slice;
    // CTAs: up to 64 slices are one cluster per block, a few slices per CTA, merged by asynchronous stores.  Measured
    // on one token through 24 layers (fp16 896 x 1152 and 896 x 896, 38 and 56 slices, int8 cache of 2001 keys, one graph):
    // a CTA per slice and a merge through the workspace 10.5 and 9.4 us per launch, 536 us per token; this and programmatic
    // launches of this kernel and the attention kernel, 229 us.  More slices (few columns, many rows) are merged
    // through the workspace.
    const bool wide = w_kind == 1 && P.n_out % 8 == 0;   // fp16 rows of whole 16-byte pieces
    if (n_slices <= PJ_CLUSTER * PJ_SLOTS) {
        P.slots = (n_slices + PJ_CLUSTER - 1) / PJ_CLUSTER;
        P.ctas = P.cl_size = (n_slices + P.slots - 1) / P.slots;
    } else {
        P.slots = wide ? 4 : 2;
        P.ctas = (n_slices + P.slots - 1) / P.slots;
        P.cl_size = 1;
        const size_t need = (size_t)n_slices * P.n_out * sizeof(float);
        MX_REQUIRE(h->ws && need <= h->ws_bytes, MX230_ERR_WORKSPACE, "%s: workspace %zu B < %zu B needed", who,
                   h->ws_bytes, need);
        MX_REQUIRE((size_t)n_blocks <= h->n_counters, MX230_ERR_UNSUPPORTED, "%s: %d column blocks exceed %zu counters",
                   who, n_blocks, h->n_counters);
        h->staged.valid = 0;   // the workspace is about to hold something else
        P.partials = (float *)h->ws;
        P.counters = h->counters;
    }
    P.status = h->status_dev;
    P.test_drop = h->test_drop_tile;
    mx230_device_guard guard(h->device);
    cudaStream_t st = (cudaStream_t)stream;
    const dim3 grid((unsigned)(n_blocks * P.ctas));
    const int threads = P.slots * PJ_ROWLANES * PJ_COLS / (wide ? 8 : 4);
    // rows/4 words + rows/ag scales; up to 12288 rows per slice fit
    const size_t sm = w_kind == 2 ? (size_t)P.slots * P.rows_per_slice * sizeof(float) / 2 : 0;
    const int cx = P.cl_size;
    if (w_kind == 2) {
        MX_SMEM_ATTR_ONCE(h->device, (gemv_heads_kernel<int8_t, 4>), 192 * 1024);
        MX_LAUNCH(h, st, MX230_K_GEMV, mx_launch(gemv_heads_kernel<int8_t, 4>, grid, threads, sm, st, cx, true, P));
    } else if (wide) MX_LAUNCH(h, st, MX230_K_GEMV, mx_launch(gemv_heads_kernel<__half, 8>, grid, threads, sm, st, cx, true, P));
    else if (w_kind == 1) MX_LAUNCH(h, st, MX230_K_GEMV, mx_launch(gemv_heads_kernel<__half, 4>, grid, threads, sm, st, cx, true, P));
    else MX_LAUNCH(h, st, MX230_K_GEMV, mx_launch(gemv_heads_kernel<float, 4>, grid, threads, sm, st, cx, true, P));
    return MX230_OK;
}

}  // namespace

extern "C" int mx230_gemv(mx230_handle *h, void *stream, float *y, const float *x, const void *w, int w_fp16,
                          const float *b, int n_in, int n_out, int accum) {
    GemvParams P{};
    P.y = y, P.x = x, P.w = w, P.b = b, P.n_in = n_in, P.n_out = n_out, P.accum = accum ? 1 : 0;
    return launch_gemv(h, stream, P, w_fp16 ? 1 : 0, "gemv");
}

extern "C" int mx230_gemv_int8(mx230_handle *h, void *stream, float *y, const float *x, const void *w_packed,
                               const float *scales, const float *b, int n_in, int n_out, int accum, int act_group) {
    GemvParams P{};
    P.y = y, P.x = x, P.w = w_packed, P.b = b, P.n_in = n_in, P.n_out = n_out, P.accum = accum ? 1 : 0;
    P.scales = scales, P.ag = act_group;
    return launch_gemv(h, stream, P, 2, "gemv_int8");
}

extern "C" int mx230_qkv_rope_kvwrite(mx230_handle *h, void *stream, float *qkv, const float *x, const void *w,
                                      int w_kind, const float *w_scales, int act_group, const float *b, int n_in,
                                      int pos, const int *pos_ptr,
                                      int n_head, int n_kv_head, int head_dim, float theta, float *kcache,
                                      float *vcache, int8_t *kq, int8_t *vq, float *ks, float *vs, float *kb,
                                      float *vb, const int *bt, int bs) {
    MX_REQUIRE(head_dim == 64, MX230_ERR_UNSUPPORTED, "qkv_rope_kvwrite: head_dim %d unsupported (must be 64)", head_dim);
    MX_REQUIRE(n_head > 0 && n_kv_head > 0, MX230_ERR_INVALID_ARG, "qkv_rope_kvwrite: bad head counts %d/%d", n_head, n_kv_head);
    MX_REQUIRE((kq != nullptr) ? (vq && ks && vs && ((kb == nullptr) == (vb == nullptr))) : (kcache && vcache),
               MX230_ERR_INVALID_ARG, "qkv_rope_kvwrite: missing cache array");
    MX_REQUIRE(pos_ptr || pos >= 0, MX230_ERR_INVALID_ARG, "qkv_rope_kvwrite: negative position %d", pos);
    MX_REQUIRE(bt == nullptr || bs > 0, MX230_ERR_INVALID_ARG, "qkv_rope_kvwrite: block size %d", bs);
    GemvParams P{};
    MX_REQUIRE(w_kind >= 0 && w_kind <= 2, MX230_ERR_INVALID_ARG, "qkv_rope_kvwrite: weight kind %d", w_kind);
    P.y = qkv, P.x = x, P.w = w, P.b = b, P.n_in = n_in, P.n_out = (n_head + 2 * n_kv_head) * 64, P.accum = 0;
    P.scales = w_scales, P.ag = act_group;
    P.e.enabled = 1, P.e.pos = pos, P.e.pos_dev = pos_ptr, P.e.n_head = n_head, P.e.n_kv_head = n_kv_head;
    P.e.theta = theta, P.e.kcache = kcache, P.e.vcache = vcache, P.e.kq = kq, P.e.vq = vq;
    P.e.ks = ks, P.e.vs = vs, P.e.kb = kb, P.e.vb = vb, P.e.bt = bt, P.e.bs = bs;
    return launch_gemv(h, stream, P, w_kind, "qkv_rope_kvwrite");
}
