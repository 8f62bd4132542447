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
// gives one thread a whole output column.  Here a 64-column block (one attention head) belongs to a thread-block cluster
// of up to eight CTAs, each with a slice of the input rows small enough that a thread's loads are all in flight at once;
// the CTAs push their 64 sums into the first one's shared memory, which adds them in slice order (deterministic), adds
// the bias and runs the epilogue.  Only matrices whose slices would get long (or that have few columns) use several
// clusters per block, merged through the workspace by the last one to arrive.  The kernel is launched programmatically:
// its slice of the weights is on its way into L2 while the kernel before it still runs.
#include <cuda_fp16.h>

#include "common.cuh"

namespace {

constexpr int PJ_THREADS = 256;
constexpr int PJ_WARPS = PJ_THREADS / 32;
constexpr int PJ_COLS = 64;     // columns per CTA = one head
constexpr int PJ_CLUSTER = 8;   // most CTAs of a column block that merge through shared memory
constexpr int PJ_MAX_ROWS = 4096;   // input rows per CTA at most (bounds the int8 path's shared memory)

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
    int rows_per_slice, n_slices, cl_size;   // n_slices = clusters per block x cl_size
    float *partials;         // [clusters per block][n_out]
    unsigned *counters;      // one per column block, self-resetting
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

// Grid: column blocks x n_slices, slices fastest; a cluster holds cl_size consecutive slices of one block.
template <typename WT, int CPT>
__global__ void __launch_bounds__(PJ_THREADS)
gemv_heads_kernel(const GemvParams P) {
    constexpr bool I8 = sizeof(WT) == 1;
    constexpr int TPR = PJ_COLS / CPT;              // threads across a weight row
    constexpr int RL = PJ_THREADS / TPR;            // weight rows per pass
    constexpr int BATCH = 4;                        // passes whose loads are issued together
    constexpr int ELT = I8 ? 4 : (int)sizeof(WT);   // bytes of a stored weight word
    constexpr int IN_PER_ROW = I8 ? 4 : 1;          // input rows in one stored row
    __shared__ float red[PJ_WARPS][PJ_COLS];
    __shared__ float parts[PJ_CLUSTER][PJ_COLS];    // first CTA of the cluster: the sums of every CTA
    __shared__ float val[PJ_COLS];
    __shared__ int is_last;
    extern __shared__ float xs[];                   // int8: this slice of x as packed codes, then group scales
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, C = P.cl_size;
    const int blk = blockIdx.x / P.n_slices, slice = blockIdx.x - blk * P.n_slices;
    const int cl = slice / C, rank = slice - cl * C;
    const int col0 = blk * PJ_COLS;
    const int k0 = min(P.n_in, slice * P.rows_per_slice), k1 = min(P.n_in, k0 + P.rows_per_slice);
    const int r0 = k0 / IN_PER_ROW, r1 = k1 / IN_PER_ROW;   // stored rows of this slice

    mx::pdl_trigger();
    if (C > 1) mx::cluster_arrive_relaxed();        // waited for before the first access to another CTA's memory
    // start of the slice into L2 under the previous kernel's tail
    for (int r = r0 + tid; r < min(r1, r0 + 2 * PJ_THREADS); r += PJ_THREADS) {
        const char *line = (const char *)P.w + ((size_t)r * P.n_out + col0) * ELT;
        mx::prefetch_l2(line);
        if (ELT == 4 && col0 + 32 < P.n_out) mx::prefetch_l2(line + 128);
    }
    mx::pdl_wait();

    const int cq = tid % TPR, rl = tid / TPR;
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
            const int i = r + u * RL;
            const bool in = live && i < r1;
            if (in) w[u].load(P.w, (size_t)i * P.n_out + col);
            else w[u].zero();
            if (!I8) xv[u] = in ? P.x[i] : 0.0f;
        }
    };
    load(r0 + rl);
    // what the epilogue of the cluster's first CTA needs, under the weight loads
    const QkvEpilogue &E = P.e;
    const bool is_v = blk >= E.n_head + E.n_kv_head;
    float bias = 0.0f, scale_o = 1.0f, y_old = 0.0f, cs = 1.0f, sn = 0.0f;
    int pos = 0;
    size_t row = 0;
    if (rank == 0 && tid < PJ_COLS && col0 + tid < P.n_out) {
        const int o = col0 + tid;
        if (P.b) bias = P.b[o];
        if (I8) scale_o = P.scales[o];
        if (P.accum) y_old = P.y[o];
        if (E.enabled && tid < 32) {
            pos = E.pos_dev ? *E.pos_dev : E.pos;
            row = E.bt && blk >= E.n_head ? (size_t)(E.bt[pos / E.bs] * E.bs + pos % E.bs) : (size_t)pos;
            if (!is_v) mx::rope_angle(pos, tid, 64, E.theta, cs, sn);
        }
    }
    if constexpr (I8) {
        // quantise this slice of the activations exactly as the reference kernel does
        const int ag = P.ag;
        int *xq = (int *)xs;                        // (k1 - k0) / 4 words
        float *xsc = xs + P.rows_per_slice / 4;     // (k1 - k0) / ag scales
        for (int g = tid; g < (k1 - k0) / ag; g += PJ_THREADS) {
            const float *xg = P.x + k0 + g * ag;
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
        for (int r = r0 + rl; r < r1; r += BATCH * RL) {
            if (r != r0 + rl) load(r);
#pragma unroll
            for (int u = 0; u < BATCH; ++u) {
                const int q = r + u * RL - r0;
                if (q < r1 - r0) w[u].fma(xq[q], xsc[q / wpg], acc);
            }
        }
    } else {
        for (int r = r0 + rl; r < r1; r += BATCH * RL) {
            if (r != r0 + rl) load(r);
#pragma unroll
            for (int u = 0; u < BATCH; ++u) w[u].fma(xv[u], acc);
        }
    }
    // ---- CTA, then cluster, then (several clusters) block totals ----
#pragma unroll
    for (int c = 0; c < CPT; ++c) {
#pragma unroll
        for (int o = TPR; o < 32; o <<= 1) acc[c] += __shfl_xor_sync(0xFFFFFFFFu, acc[c], o);
        if (lane < TPR) red[warp][CPT * cq + c] = acc[c];
    }
    __syncthreads();
    float sum = 0.0f;
    if (tid < PJ_COLS) {
#pragma unroll
        for (int r = 0; r < PJ_WARPS; ++r) sum += red[r][tid];
    }
    if (C > 1) {
        mx::cluster_wait();       // every CTA of the cluster runs
        if (tid < PJ_COLS) mx::cluster_st_f32(mx::cluster_map(mx::smem_u32(&parts[rank][tid]), 0), sum);
        mx::cluster_sync();
        if (rank != 0) return;
        if (tid < PJ_COLS) {
            sum = 0.0f;
            for (int r = 0; r < C; ++r) sum += parts[r][tid];
        }
    }
    const int n_cl = P.n_slices / C;
    if (n_cl > 1) {
        if (tid < PJ_COLS && col0 + tid < P.n_out) P.partials[(size_t)cl * P.n_out + col0 + tid] = sum;
        __threadfence();
        __syncthreads();
        if (tid == 0) is_last = atomicInc(&P.counters[blk], n_cl - 1) == (unsigned)(n_cl - 1);
        __syncthreads();
        if (!is_last) return;
        __threadfence();
        if (tid < PJ_COLS && col0 + tid < P.n_out) {
            sum = 0.0f;
            for (int r = 0; r < n_cl; ++r) sum += __ldcg(P.partials + (size_t)r * P.n_out + col0 + tid);
        }
    }
    // ---- epilogue on the 64 finished sums of this column block ----
    if (tid < PJ_COLS) val[tid] = (I8 ? sum * scale_o : sum) + bias;
    __syncthreads();
    if (!E.enabled) {
        if (tid < PJ_COLS && col0 + tid < P.n_out) P.y[col0 + tid] = P.accum ? y_old + val[tid] : val[tid];
        return;
    }
    // qkv step: this block is head `hb` of the row [Q heads | K heads | V heads]
    const int hb = blk;
    if (tid < 32) {   // one warp: lane l owns the rotation pair (l, l + 32), then elements 2l, 2l+1
        if (!is_v) mx::rope_pair(val[tid], val[tid + 32], cs, sn);
        __syncwarp();
        const float2 x2 = make_float2(val[2 * tid], val[2 * tid + 1]);
        *(float2 *)(P.y + (size_t)hb * 64 + 2 * tid) = x2;
        if (hb >= E.n_head) {   // K or V head: the cache row of this position
            const int kvh = is_v ? hb - E.n_head - E.n_kv_head : hb - E.n_head;
            const int kvd = E.n_kv_head * 64;
            if (E.kq == nullptr) {
                float *dst = (is_v ? E.vcache : E.kcache) + row * kvd + kvh * 64;
                *(float2 *)(dst + 2 * tid) = x2;
            } else {
                int8_t *dst = (is_v ? E.vq : E.kq) + row * kvd + kvh * 64;
                float *sc = is_v ? E.vs : E.ks, *be = is_v ? E.vb : E.kb;
                const size_t sd = row * E.n_kv_head + kvh;
                int c0, c1;
                float scale, beta;
                mx::quant_head_row(x2.x, x2.y, be != nullptr, c0, c1, scale, beta);
                if (tid == 0) {
                    sc[sd] = scale;
                    if (be != nullptr) be[sd] = beta;
                }
                *(unsigned short *)(dst + 2 * tid) = (unsigned short)((c0 & 0xFF) | ((c1 & 0xFF) << 8));
            }
        }
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
    const bool wide = w_kind == 1 && P.n_out % 8 == 0;   // fp16 rows of whole 16-byte pieces
    const int pass = (wide ? 32 : 16) * (w_kind == 2 ? 4 : 1);   // input rows that a CTA takes in one load per thread
    // Measured on one token through 24 layers (fp16 896 x 1152 and 896 x 896, int8 cache of 2001 keys, one graph): with 38 and
    // 56 slices merged through the workspace 10.5 and 9.4 us per launch, 536 us per token; one cluster of eight per block
    // and programmatic launches of this kernel and the attention kernel, 247 us.
    // One cluster per column block, of as many CTAs (up to 8) as have a pass of rows each.  Further clusters (a merge
    // through global memory, about 2 us) only where the blocks alone leave SMs idle and every CTA still gets four passes,
    // or where a slice would exceed PJ_MAX_ROWS.
    int c = (P.n_in + pass - 1) / pass;
    P.cl_size = c < PJ_CLUSTER ? c : PJ_CLUSTER;
    long long n_cl = (2ll * h->sm_count + n_blocks * P.cl_size - 1) / ((long long)n_blocks * P.cl_size);
    const long long by_rows = P.n_in / ((long long)P.cl_size * 4 * pass);
    if (n_cl > by_rows) n_cl = by_rows;
    const long long at_least = (P.n_in + (long long)P.cl_size * PJ_MAX_ROWS - 1) / ((long long)P.cl_size * PJ_MAX_ROWS);
    if (n_cl < at_least) n_cl = at_least;
    P.n_slices = (int)n_cl * P.cl_size;
    const int gran = w_kind == 2 ? 8 : 1;   // int8: a slice holds whole activation groups
    P.rows_per_slice = ((P.n_in + P.n_slices - 1) / P.n_slices + gran - 1) / gran * gran;
    if (n_cl > 1) {
        const size_t need = (size_t)n_cl * P.n_out * sizeof(float);
        MX_REQUIRE(h->ws && need <= h->ws_bytes, MX230_ERR_WORKSPACE, "%s: workspace %zu B < %zu B needed", who,
                   h->ws_bytes, need);
        MX_REQUIRE((size_t)n_blocks <= h->n_counters, MX230_ERR_UNSUPPORTED, "%s: %d column blocks exceed %zu counters",
                   who, n_blocks, h->n_counters);
        h->staged.valid = 0;   // the workspace is about to hold something else
        P.partials = (float *)h->ws;
        P.counters = h->counters;
    }
    mx230_device_guard guard(h->device);
    cudaStream_t st = (cudaStream_t)stream;
    const dim3 grid((unsigned)(n_blocks * P.n_slices));
    const size_t sm = w_kind == 2 ? (size_t)P.rows_per_slice * sizeof(float) / 2 : 0;   // rows/4 words + rows/ag scales
    const int cx = P.cl_size;
    if (w_kind == 2) MX_LAUNCH(h, st, MX230_K_GEMV, mx_launch(gemv_heads_kernel<int8_t, 4>, grid, PJ_THREADS, sm, st, cx, true, P));
    else if (wide) MX_LAUNCH(h, st, MX230_K_GEMV, mx_launch(gemv_heads_kernel<__half, 8>, grid, PJ_THREADS, sm, st, cx, true, P));
    else if (w_kind == 1) MX_LAUNCH(h, st, MX230_K_GEMV, mx_launch(gemv_heads_kernel<__half, 4>, grid, PJ_THREADS, sm, st, cx, true, P));
    else MX_LAUNCH(h, st, MX230_K_GEMV, mx_launch(gemv_heads_kernel<float, 4>, grid, PJ_THREADS, sm, st, cx, true, P));
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
