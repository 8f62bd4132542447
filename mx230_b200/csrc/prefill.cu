// Per-layer attention step, part 3: prefill attention of n_tok new rows at absolute
// positions pos0+qi over the KV cache (keys 0..=pos0+qi), grouped-query aware.
//
// Reference semantics: attn_prefill_body<KIND, PAGED> and its wrappers,
// 03-llm-engine/kernels/llm.cu:3657-3872 -- a flash-style fp32 SIMT kernel per
// (64-query tile, head) that reads q strided from the qkv buffer and K/V only from the
// cache (so under an int8 cache a token attends the *quantised* K/V of itself and of
// its batch-mates, exactly as decode does).
//
// This design: one staging kernel, then the tensor-core flash kernel of the stage-2 forward with the GQA head mapping (K/V
// head = h / group), the causal offset pos0 and the reference's strided output layout.  The staging kernel brings the
// operands into that kernel's bf16 head-major layout (Q gathered from the strided qkv rows, K and V from the cache through
// the optional block table) and, in the prefill step, does the work in front of attention in the same pass: RoPE on the
// new rows, their K and V written to the cache (fp32 copy or int8 quantize-on-write) and staged from registers.
// KIND 2 of the reference (scores through on-the-fly int8 K, an opt-in speed approximation on sm_61) is served over an
// fp32 cache by quantising K while it is staged.
#include "common.cuh"

namespace {

constexpr int HD = 64;

struct StageParams {
    // operands of the attention kernel
    __nv_bfloat16 *qout;             // [n_head][n_tok][64]
    __nv_bfloat16 *kout, *vout;      // [n_kv_head][n_keys][64]
    float *q_norm2, *k_norm2;        // [heads][MX230_NORM_PARTS] largest squared norm of the (dequantised) rows of each part, or null
    float *row_a, *row_qsum, *kskb;  // int8 scores: per-row factor and code sum; per-key scale and offset by tiles of 128
    int n_k_tiles;
    // inputs
    float *qkv;
    int stride, n_tok, pos0, n_keys, n_head, n_kv_head;
    float *kcache, *vcache;          // fp32 cache, or
    int8_t *kq, *vq;                 // int8 cache with
    float *ks, *vs, *kb, *vb;        // per-(row, head) scale and (optional) beta
    const int *bt;
    int bs;
    // the step's work in front of attention
    int old_warps;                   // warps of a CTA that take cached keys, from the last one on
    int write_kv;                    // the new rows' K and V come from qkv and go to the cache (else they are in it)
    int rope;
    float theta;
};

constexpr int ST_THREADS = 512;
constexpr int ST_WARPS = ST_THREADS / 32;
constexpr int ST_SUBS = 4;           // warps that share a token (they take its heads in turn)
constexpr int ST_HEADS = 5;          // heads of a warp whose loads are issued together (14 + 2 * 2 heads: one round)

__device__ __forceinline__ size_t stage_row(const StageParams &P, int t) {
    return P.bt ? (size_t)(P.bt[t / P.bs] * P.bs + t % P.bs) : (size_t)t;
}
__device__ __forceinline__ float *stage_kskb(const StageParams &P, int h, int t) {
    return P.kskb + ((size_t)h * P.n_k_tiles + (t >> 7)) * 256 + (t & 127);
}

// 128 or 256 CTAs whatever the size: the kernel is a few microseconds of latency (launch, one or two memory round trips), so
// what counts is that it is ONE launch and that every thread's loads are issued together.  In its place stood rope 5.4 us,
// quantise 4, two staging kernels 3.8 + 4 (512 tokens over 1536 cached keys, int8), and 11.7 + 5 + 4.7 + 5 (1900 tokens,
// fp32).  New tokens: four warps per token, lane l holds dims l and l + 32 of a head, so RoPE's angle is computed once
// per token and warp and a head's quantiser is a warp reduction.  Cached keys: eight threads per key and head, eight dims
// each.  What a warp of new tokens costs is the code it fetches as much as its arithmetic: its heads are one rolled loop over
// values in shared memory, an instantiation per cache and score mode, and the first angle is formed before the wait (512 tokens over
// 1536 int8 keys, from the wait to the last token 4.3 -> 4.1 us and to the norms 5.9 -> 5.0, a call 26.9 -> 24.6; over fp32 keys 20.4 -> 19.0).  Row norms go through shared memory and, per cluster of CTAs, into one of MX230_NORM_PARTS parts: with Q's
// and K's the attention kernel bounds every score of a head and, where the bound is small, runs without a row max.
// CLUSTER: CTAs that share one norm part, 4 or 8.  I8: int8 scores; Q8: int8 cache (instantiations: code that a launch does not
// run is not fetched either).  (Sizes are constants or come from the host: a division costs more here than
// the work of a thread.)
template <int CLUSTER, bool I8, bool Q8>
__global__ void __launch_bounds__(ST_THREADS, 2) prefill_stage_kernel(const StageParams P) {
    extern __shared__ float2 heads[];   // [ST_WARPS][ST_HEADS][32] a warp's heads of its token: lane l's dims l and l + 32
    int *smax = (int *)(heads + ST_WARPS * ST_HEADS * 32);   // [n_norms] squared norms of Q and K heads as ordered integers (NaN largest)
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int n_ctas = MX230_NORM_PARTS * CLUSTER;
    const int n_max = P.n_head + P.n_kv_head, n_norms = P.q_norm2 ? n_max : 0;
    mx::pdl_trigger();
    for (int i = tid; i < n_norms; i += ST_THREADS) smax[i] = 0;
    __syncthreads();
    mx::cluster_arrive_release();    // waited for before this CTA adds to the first one's maxima
    const int sub = warp & (ST_SUBS - 1), tok0 = blockIdx.x + n_ctas * (warp / ST_SUBS);
    float cs = 1.0f, sn = 0.0f;      // of the warp's next token; its first one's before the wait: the angle takes as long as a load
    if (P.rope && tok0 < P.n_tok) mx::rope_angle(P.pos0 + tok0, lane, HD, P.theta, cs, sn);
    mx::pdl_wait();
    auto raise = [&](int head, float norm2) {
        if (n_norms > 0) atomicMax(&smax[head], __float_as_int(norm2) & 0x7FFFFFFF);
    };
    const size_t kvd = (size_t)P.n_kv_head * HD;

    // ---- new tokens ----
    const int n_units = P.n_head + (P.write_kv ? 2 * P.n_kv_head : 0);
    float va[ST_HEADS], vb[ST_HEADS];
    auto load = [&](int tok, int u0) {
        const float *row = P.qkv + (size_t)tok * P.stride;
#pragma unroll
        for (int i = 0; i < ST_HEADS; ++i) {
            const int u = u0 + i * ST_SUBS;
            if (u < n_units) va[i] = row[u * HD + lane], vb[i] = row[u * HD + 32 + lane];
        }
    };
    if (tok0 < P.n_tok) load(tok0, sub);
    for (int tok = tok0, u0 = sub; tok < P.n_tok;) {
        const int pos = P.pos0 + tok;
        float *row = P.qkv + (size_t)tok * P.stride;
        const size_t crow = P.write_kv ? stage_row(P, pos) : 0;
#pragma unroll
        for (int i = 0; i < ST_HEADS; ++i) heads[(warp * ST_HEADS + i) * 32 + lane] = make_float2(va[i], vb[i]);
        // the warp's next heads, of this token or of its next, arrive under these
        int next = tok, next_u0 = u0 + ST_HEADS * ST_SUBS;
        if (next_u0 >= n_units) next += n_ctas * (ST_WARPS / ST_SUBS), next_u0 = sub;
        if (next < P.n_tok) load(next, next_u0);
        // (a lane reads what it wrote.  Not unrolled: with five copies of the loop, code for the instruction cache, 0.7 us slower)
#pragma unroll 1
        for (int i = 0; i < ST_HEADS; ++i) {
            const int u = u0 + i * ST_SUBS;
            if (u >= n_units) break;
            const float2 ab = heads[(warp * ST_HEADS + i) * 32 + lane];
            float a = ab.x, b = ab.y;
            if (P.rope && u < n_max) {   // Q and K heads
                mx::rope_pair(a, b, cs, sn);
                row[u * HD + lane] = a, row[u * HD + 32 + lane] = b;
            }
            float hi = 0.0f, lo = 0.0f;   // range of the head's values, for the quantisers
            if (I8 || Q8) hi = mx::warp_max(fmaxf(a, b)), lo = mx::warp_min(fminf(a, b));
            if (u < P.n_head) {
                __nv_bfloat16 *dst = P.qout + ((size_t)u * P.n_tok + tok) * HD;
                if (I8) {
                    // q row -> int8 codes per (row, head): id = 127 / amax, code = clamp(rne(q * id), +-127); the
                    // codes go out as bf16 (exact), with the row's score factor (amax / 127) * 1/sqrt(64) * log2(e)
                    // and the sum of its codes (the reference's own arithmetic, llm.cu:3700-3716)
                    const float amax = fmaxf(fabsf(hi), fabsf(lo));
                    const float id = amax > 0.0f ? __fdiv_rn(127.0f, amax) : 0.0f;
                    const int ca = max(-127, min(127, __float2int_rn(a * id))), cb = max(-127, min(127, __float2int_rn(b * id)));
                    const int sum = __reduce_add_sync(0xFFFFFFFFu, ca + cb), sq = __reduce_add_sync(0xFFFFFFFFu, ca * ca + cb * cb);
                    dst[lane] = __float2bfloat16((float)ca);
                    dst[lane + 32] = __float2bfloat16((float)cb);
                    if (lane == 0) {
                        const float qs = amax > 0.0f ? __fdiv_rn(amax, 127.0f) : 0.0f;
                        P.row_a[(size_t)u * P.n_tok + tok] = qs * 0.125f * 1.4426950408889634f;
                        P.row_qsum[(size_t)u * P.n_tok + tok] = (float)sum;
                        raise(u, qs * qs * (float)sq);
                    }
                } else {
                    // values times 1/sqrt(64) * log2(e), one rounding: the scores arrive in log2 units
                    dst[lane] = __float2bfloat16_rn(a * MX230_QK_LOG2_SCALE);
                    dst[lane + 32] = __float2bfloat16_rn(b * MX230_QK_LOG2_SCALE);
                    float ss = a * a + b * b;
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xFFFFFFFFu, ss, o);
                    if (lane == 0) raise(u, ss);
                }
                continue;
            }
            const bool is_v = u >= n_max;
            const int h = is_v ? u - n_max : u - P.n_head;
            __nv_bfloat16 *dst = (is_v ? P.vout : P.kout) + ((size_t)h * P.n_keys + pos) * HD;
            float x0 = a, x1 = b;   // what attention sees
            if (Q8) {
                int8_t *cdst = (is_v ? P.vq : P.kq) + crow * kvd + h * HD;
                float *sc = is_v ? P.vs : P.ks, *be = is_v ? P.vb : P.kb;
                int c0, c1;
                float scale, beta;
                mx::quant_head_row(a, b, hi, lo, be != nullptr, c0, c1, scale, beta);
                cdst[lane] = (int8_t)c0, cdst[lane + 32] = (int8_t)c1;
                if (lane == 0) {
                    sc[crow * P.n_kv_head + h] = scale;
                    if (be) be[crow * P.n_kv_head + h] = beta;
                }
                x0 = (float)c0 * scale + beta, x1 = (float)c1 * scale + beta;
                a = x0, b = x1;
                if (I8 && !is_v) {
                    x0 = (float)c0, x1 = (float)c1;
                    if (lane == 0) {
                        float *kk = stage_kskb(P, h, pos);
                        kk[0] = scale, kk[128] = beta;
                    }
                }
            } else {
                float *cdst = (is_v ? P.vcache : P.kcache) + crow * kvd + h * HD;
                cdst[lane] = a, cdst[lane + 32] = b;
            }
            dst[lane] = __float2bfloat16_rn(x0);
            dst[lane + 32] = __float2bfloat16_rn(x1);
            if (!is_v) {
                float ss = a * a + b * b;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xFFFFFFFFu, ss, o);
                if (lane == 0) raise(P.n_head + h, ss);
            }
        }
        if (next != tok && next < P.n_tok && P.rope) mx::rope_angle(P.pos0 + next, lane, HD, P.theta, cs, sn);
        tok = next, u0 = next_u0;
    }

    // ---- cached keys [0, n_old): from the last warp of every CTA on, the first ones have the new tokens ----
    const int n_old = P.write_kv ? P.pos0 : P.n_keys;
    const size_t total = (size_t)n_old * P.n_kv_head * 8;
    const int W = P.old_warps;
    for (size_t base = (blockIdx.x * (size_t)W + (ST_WARPS - 1 - warp)) * 32; ST_WARPS - 1 - warp < W && base < total;
         base += (size_t)n_ctas * W * 32) {
        const bool live = base + lane < total;
        const size_t idx = live ? base + lane : total - 1;   // keep the row's lanes together for the shuffles below
        const int c = (int)(idx & 7);
        const size_t th = idx >> 3;
        const int t = total >> 32 ? (int)(th / P.n_kv_head) : (int)((uint32_t)th / (uint32_t)P.n_kv_head);
        const int h = (int)(th - (size_t)t * P.n_kv_head);
        const size_t row = stage_row(P, t);
        const size_t dst = ((size_t)h * P.n_keys + t) * HD + c * 8;
        float k[8], v[8], ksc = 0.0f, kbe = 0.0f, ss = 0.0f;
        if (Q8) {
            const int2 kw = *(const int2 *)(P.kq + row * kvd + h * HD + c * 8);
            const int2 vw = *(const int2 *)(P.vq + row * kvd + h * HD + c * 8);
            ksc = P.ks[row * P.n_kv_head + h];
            kbe = P.kb ? P.kb[row * P.n_kv_head + h] : 0.0f;
            const float vsc = P.vs[row * P.n_kv_head + h], vbe = P.vb ? P.vb[row * P.n_kv_head + h] : 0.0f;
            const int kk[2] = {kw.x, kw.y}, vv[2] = {vw.x, vw.y};
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                // dequantise as the reference does into its V tile: code * scale + beta (llm.cu:3759-3764)
                const float code = (float)(int8_t)((kk[i >> 2] >> (8 * (i & 3))) & 0xFF);
                const float val = code * ksc + kbe;
                ss += val * val;
                k[i] = I8 ? code : val;
                v[i] = (float)(int8_t)((vv[i >> 2] >> (8 * (i & 3))) & 0xFF) * vsc + vbe;
            }
        } else {
            const float4 *kp = (const float4 *)(P.kcache + row * kvd + h * HD + c * 8);
            const float4 *vp = (const float4 *)(P.vcache + row * kvd + h * HD + c * 8);
            const float4 a = kp[0], b = kp[1], e = vp[0], f = vp[1];
            k[0] = a.x, k[1] = a.y, k[2] = a.z, k[3] = a.w, k[4] = b.x, k[5] = b.y, k[6] = b.z, k[7] = b.w;
            v[0] = e.x, v[1] = e.y, v[2] = e.z, v[3] = e.w, v[4] = f.x, v[5] = f.y, v[6] = f.z, v[7] = f.w;
            if (I8) {   // K quantised on the fly, symmetric absmax per row (the reference's attn_prefill_dp4a)
                float amax = 0.0f;
#pragma unroll
                for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(k[i]));
#pragma unroll
                for (int o = 4; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, o));
                const float id = amax > 0.0f ? __fdiv_rn(127.0f, amax) : 0.0f;
                ksc = amax > 0.0f ? __fdiv_rn(amax, 127.0f) : 0.0f;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    k[i] = (float)max(-127, min(127, __float2int_rn(k[i] * id)));
                    ss += k[i] * ksc * (k[i] * ksc);
                }
            } else {
#pragma unroll
                for (int i = 0; i < 8; ++i) ss += k[i] * k[i];
            }
        }
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) ss += __shfl_xor_sync(0xFFFFFFFFu, ss, o);   // the row's eight threads
        if (!live) continue;
        uint4 ko, vo;
        ko.x = mx::pack_bf16(k[0], k[1]), ko.y = mx::pack_bf16(k[2], k[3]);
        ko.z = mx::pack_bf16(k[4], k[5]), ko.w = mx::pack_bf16(k[6], k[7]);
        vo.x = mx::pack_bf16(v[0], v[1]), vo.y = mx::pack_bf16(v[2], v[3]);
        vo.z = mx::pack_bf16(v[4], v[5]), vo.w = mx::pack_bf16(v[6], v[7]);
        *(uint4 *)(P.kout + dst) = ko;
        *(uint4 *)(P.vout + dst) = vo;
        if (c == 0) {
            if (I8) {
                float *kk = stage_kskb(P, h, t);
                kk[0] = ksc, kk[128] = kbe;
            }
            raise(P.n_head + h, ss);
        }
    }

    // ---- the cluster's maxima -> its part ----
    const int part = blockIdx.x / CLUSTER, rank = blockIdx.x % CLUSTER;
    __syncthreads();
    mx::cluster_wait();
    if (rank != 0)
        for (int i = tid; i < n_norms; i += ST_THREADS) mx::cluster_red_max(mx::cluster_map(mx::smem_u32(&smax[i]), 0), smax[i]);
    mx::cluster_sync();
    if (rank != 0) return;
    for (int i = tid; i < n_norms; i += ST_THREADS) {
        float *dst = i < P.n_head ? P.q_norm2 + (size_t)i * MX230_NORM_PARTS : P.k_norm2 + (size_t)(i - P.n_head) * MX230_NORM_PARTS;
        dst[part] = __int_as_float(smax[i]);
    }
}

// What the prefill step adds to plain prefill attention
struct StepArgs {
    bool write_kv;
    int rope;
    float theta;
};

// sm: bytes of the norms
constexpr size_t ST_NORM_BYTES = 48 * 1024, ST_HEAD_BYTES = (size_t)ST_WARPS * ST_HEADS * 64 * sizeof(float);
template <bool I8, bool Q8>
int launch_stage(mx230_handle *h, cudaStream_t st, const StageParams &S, int cluster, size_t sm) {
    MX_SMEM_ATTR_ONCE(h->device, (prefill_stage_kernel<4, I8, Q8>), ST_HEAD_BYTES + ST_NORM_BYTES);
    MX_SMEM_ATTR_ONCE(h->device, (prefill_stage_kernel<8, I8, Q8>), ST_HEAD_BYTES + ST_NORM_BYTES);
    MX_LAUNCH(h, st, MX230_K_PREFILL,
              mx_launch(cluster == 8 ? prefill_stage_kernel<8, I8, Q8> : prefill_stage_kernel<4, I8, Q8>, MX230_NORM_PARTS * cluster, ST_THREADS,
                        ST_HEAD_BYTES + sm, st, cluster, true, S));
    return MX230_OK;
}

size_t align1k(size_t x) { return (x + 1023) & ~(size_t)1023; }

// With a step, qkv and the cache are written as well (the entry point that asks for one takes them non-const).  o_half (may be
// null) receives where the output lies in fp16, by heads: in the workspace, in Q's place.
int prefill(mx230_handle *h, void *stream, float *out, const float *qkv, const float *kcache,
            const float *vcache, const int8_t *kq, const int8_t *vq, const float *ks, const float *vs,
            const float *kb, const float *vb, int pos0, int n_tok, int n_head, int n_kv_head, int qkv_stride,
            int out_stride, const int *bt, int bs, const char *who, bool dp4a = false, StepArgs step = {}, void **o_half = nullptr) {
    MX_REQUIRE(h != nullptr, MX230_ERR_INVALID_ARG, "%s: null handle", who);
    MX_REQUIRE(pos0 >= 0 && n_tok >= 0, MX230_ERR_INVALID_ARG, "%s: negative pos0/n_tok", who);
    if (n_tok == 0) return MX230_OK;
    MX_REQUIRE(out && qkv, MX230_ERR_INVALID_ARG, "%s: null out/qkv", who);
    MX_REQUIRE(n_head > 0 && n_kv_head > 0 && n_head % n_kv_head == 0, MX230_ERR_UNSUPPORTED,
               "%s: n_head %d must be a positive multiple of n_kv_head %d", who, n_head, n_kv_head);
    if (kq)
        MX_REQUIRE(vq && ks && vs && ((kb == nullptr) == (vb == nullptr)), MX230_ERR_INVALID_ARG,
                   "%s: missing int8 cache array", who);
    else
        MX_REQUIRE(kcache && vcache, MX230_ERR_INVALID_ARG, "%s: null cache", who);
    MX_REQUIRE(bt == nullptr || bs > 0, MX230_ERR_INVALID_ARG, "%s: block size %d", who, bs);
    MX_REQUIRE(qkv_stride % 4 == 0 && out_stride % 4 == 0 &&
                   (((uintptr_t)qkv | (uintptr_t)out | (uintptr_t)kcache | (uintptr_t)vcache | (uintptr_t)kq |
                     (uintptr_t)vq) & 15) == 0,
               MX230_ERR_INVALID_ARG, "%s: buffers must be 16-byte aligned, strides multiples of 4", who);
    const int n_keys = pos0 + n_tok;
    const int n_k_pad = (n_keys + 127) / 128 * 128;
    size_t qbytes = align1k((size_t)n_head * n_tok * HD * 2);
    size_t kbytes = align1k((size_t)n_kv_head * n_keys * HD * 2);
    size_t rbytes = align1k((size_t)n_head * n_tok * 4);
    size_t cbytes = align1k((size_t)n_kv_head * n_k_pad * 8);
    size_t nbytes = align1k((size_t)(n_head + n_kv_head) * MX230_NORM_PARTS * 4);
    size_t need = qbytes + 2 * kbytes + 2 * rbytes + cbytes + nbytes;
    MX_REQUIRE(h->ws && need <= h->ws_bytes, MX230_ERR_WORKSPACE,
               "%s: workspace %zu B < %zu B needed (call mx230_reserve)", who, h->ws_bytes, need);
    mx230_device_guard guard(h->device);
    cudaStream_t st = (cudaStream_t)stream;
    h->staged.valid = 0;   // the workspace is about to hold something else
    __nv_bfloat16 *qb = (__nv_bfloat16 *)h->ws;
    if (o_half) *o_half = qb;
    __nv_bfloat16 *kbuf = (__nv_bfloat16 *)((char *)h->ws + qbytes);
    __nv_bfloat16 *vbuf = (__nv_bfloat16 *)((char *)h->ws + qbytes + kbytes);
    float *row_a = (float *)((char *)h->ws + qbytes + 2 * kbytes);
    float *row_qsum = (float *)((char *)row_a + rbytes);
    float *kskb = (float *)((char *)row_qsum + rbytes);
    float *q_norm2 = (float *)((char *)kskb + cbytes);
    float *k_norm2 = q_norm2 + (size_t)n_head * MX230_NORM_PARTS;
    // Which score arithmetic: over an int8 cache the handle's MX230_OPT_Q8_SCORE_MODE decides, as for decode
    // (REF, the default: q quantised per (row, head) to int8 and integer dots, what attn_prefill_q8 computes;
    // EXACT: fp32 q against dequantised K); the _dp4a entry points are the reference's int8-score approximation
    // over an fp32 cache by definition.
    const bool i8_scores = dp4a || (kq && h->q8_score_mode == MX230_Q8_SCORE_REF);
    StageParams S;
    S.qout = qb, S.kout = kbuf, S.vout = vbuf, S.q_norm2 = q_norm2, S.k_norm2 = k_norm2;
    S.row_a = row_a, S.row_qsum = row_qsum, S.kskb = kskb, S.n_k_tiles = n_k_pad / 128;
    S.qkv = const_cast<float *>(qkv), S.stride = qkv_stride, S.n_tok = n_tok, S.pos0 = pos0, S.n_keys = n_keys;
    S.n_head = n_head, S.n_kv_head = n_kv_head;
    S.kcache = const_cast<float *>(kcache), S.vcache = const_cast<float *>(vcache);
    S.kq = const_cast<int8_t *>(kq), S.vq = const_cast<int8_t *>(vq);
    S.ks = const_cast<float *>(ks), S.vs = const_cast<float *>(vs), S.kb = const_cast<float *>(kb), S.vb = const_cast<float *>(vb);
    S.bt = bt, S.bs = bs;
    S.write_kv = step.write_kv, S.rope = step.rope, S.theta = step.theta;
    size_t sm = (size_t)(n_head + n_kv_head) * sizeof(int);
    if (sm > ST_NORM_BYTES) {   // more heads than a CTA keeps norms for: without them every head takes the general loop
        sm = 0;
        S.q_norm2 = S.k_norm2 = q_norm2 = k_norm2 = nullptr;
    }
    // 256 CTAs, two per SM, where the warps of 128 would take tokens and cached keys in more than one round (2048 tokens over 6144
    // int8 keys, 32/4 heads, us a call: 128 176.6, 256 168.7; 512 over 1536, 14/2 heads, whose 128 CTAs have 16 warps of tokens
    // and 6 of keys, 5.1 us from the wait to their end against 1.7); below that 128, the smaller launch
    const size_t old = (size_t)(step.write_kv ? pos0 : n_keys) * n_kv_head * 8;   // threads
    auto warps_of = [&](int ctas) { return (old + 32 * ctas - 1) / (32 * ctas); };   // of a CTA, for cached keys
    const int c4 = 4 * MX230_NORM_PARTS;
    const int cluster = (size_t)((n_tok + c4 - 1) / c4) * ST_SUBS + warps_of(c4) > ST_WARPS ? 8 : 4;
    const size_t per_cta = warps_of(cluster * MX230_NORM_PARTS);
    S.old_warps = per_cta < ST_WARPS ? (int)per_cta : ST_WARPS;
    int rc;
    if (kq) rc = i8_scores ? launch_stage<true, true>(h, st, S, cluster, sm) : launch_stage<false, true>(h, st, S, cluster, sm);
    else rc = i8_scores ? launch_stage<true, false>(h, st, S, cluster, sm) : launch_stage<false, false>(h, st, S, cluster, sm);
    if (rc) return rc;
    return mx230_launch_flash_fwd_ex(h, st, qb, kbuf, vbuf, out, nullptr, n_head, n_tok, n_keys, pos0, n_head / n_kv_head, HD,
                                     out_stride, 1, i8_scores ? 0 : 1, q_norm2, k_norm2, i8_scores ? row_a : nullptr,
                                     i8_scores ? row_qsum : nullptr, i8_scores ? kskb : nullptr, o_half ? qb : nullptr);
}

}  // namespace

extern "C" size_t mx230_prefill_workspace_bytes(int n_tok, int n_keys, int n_head, int n_kv_head) {
    if (n_tok <= 0 || n_keys <= 0 || n_head <= 0 || n_kv_head <= 0) return 0;
    // staged bf16 Q, K, V, then (int8 score mode) the per-row q factors and the per-key (scale, offset) pairs
    return align1k((size_t)n_head * n_tok * HD * 2) + 2 * align1k((size_t)n_kv_head * n_keys * HD * 2) +
           2 * align1k((size_t)n_head * n_tok * 4) + align1k((size_t)n_kv_head * ((n_keys + 127) / 128 * 128) * 8) +
           align1k((size_t)(n_head + n_kv_head) * MX230_NORM_PARTS * 4);
}

extern "C" int mx230_attn_prefill(mx230_handle *h, void *stream, float *out, const float *qkv,
                                  const float *kcache, const float *vcache, int pos0, int n_tok, int n_head,
                                  int n_kv_head, int qkv_stride, int out_stride) {
    return prefill(h, stream, out, qkv, kcache, vcache, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr,
                   pos0, n_tok, n_head, n_kv_head, qkv_stride, out_stride, nullptr, 0, "attn_prefill");
}
extern "C" int mx230_attn_prefill_paged(mx230_handle *h, void *stream, float *out, const float *qkv,
                                        const float *kcache, const float *vcache, int pos0, int n_tok,
                                        int n_head, int n_kv_head, int qkv_stride, int out_stride,
                                        const int *bt, int bs) {
    MX_REQUIRE(bt, MX230_ERR_INVALID_ARG, "attn_prefill_paged: null block table");
    return prefill(h, stream, out, qkv, kcache, vcache, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr,
                   pos0, n_tok, n_head, n_kv_head, qkv_stride, out_stride, bt, bs, "attn_prefill_paged");
}
extern "C" int mx230_attn_prefill_q8(mx230_handle *h, void *stream, float *out, const float *qkv,
                                     const int8_t *kq, const int8_t *vq, const float *ks, const float *vs,
                                     const float *kb, const float *vb, int pos0, int n_tok, int n_head,
                                     int n_kv_head, int qkv_stride, int out_stride) {
    MX_REQUIRE(kq, MX230_ERR_INVALID_ARG, "attn_prefill_q8: null kq");
    return prefill(h, stream, out, qkv, nullptr, nullptr, kq, vq, ks, vs, kb, vb, pos0, n_tok, n_head,
                   n_kv_head, qkv_stride, out_stride, nullptr, 0, "attn_prefill_q8");
}
extern "C" int mx230_attn_prefill_q8_paged(mx230_handle *h, void *stream, float *out, const float *qkv,
                                           const int8_t *kq, const int8_t *vq, const float *ks,
                                           const float *vs, const float *kb, const float *vb, int pos0,
                                           int n_tok, int n_head, int n_kv_head, int qkv_stride,
                                           int out_stride, const int *bt, int bs) {
    MX_REQUIRE(kq && bt, MX230_ERR_INVALID_ARG, "attn_prefill_q8_paged: null argument");
    return prefill(h, stream, out, qkv, nullptr, nullptr, kq, vq, ks, vs, kb, vb, pos0, n_tok, n_head,
                   n_kv_head, qkv_stride, out_stride, bt, bs, "attn_prefill_q8_paged");
}
extern "C" int mx230_attn_prefill_dp4a(mx230_handle *h, void *stream, float *out, const float *qkv,
                                       const float *kcache, const float *vcache, int pos0, int n_tok,
                                       int n_head, int n_kv_head, int qkv_stride, int out_stride) {
    return prefill(h, stream, out, qkv, kcache, vcache, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr,
                   pos0, n_tok, n_head, n_kv_head, qkv_stride, out_stride, nullptr, 0, "attn_prefill_dp4a", true);
}
extern "C" int mx230_attn_prefill_dp4a_paged(mx230_handle *h, void *stream, float *out, const float *qkv,
                                             const float *kcache, const float *vcache, int pos0, int n_tok,
                                             int n_head, int n_kv_head, int qkv_stride, int out_stride,
                                             const int *bt, int bs) {
    MX_REQUIRE(bt, MX230_ERR_INVALID_ARG, "attn_prefill_dp4a_paged: null block table");
    return prefill(h, stream, out, qkv, kcache, vcache, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr,
                   pos0, n_tok, n_head, n_kv_head, qkv_stride, out_stride, bt, bs, "attn_prefill_dp4a_paged", true);
}

extern "C" int mx230_prefill_step(mx230_handle *h, void *stream, float *out, float *qkv, float *kcache, float *vcache,
                                  int8_t *kq, int8_t *vq, float *ks, float *vs, float *kb, float *vb, int pos0, int n_tok,
                                  int n_head, int n_kv_head, int head_dim, int use_rope, float theta, int qkv_stride,
                                  int out_stride, const int *bt, int bs) {
    MX_REQUIRE(head_dim == HD, MX230_ERR_UNSUPPORTED, "prefill_step: head_dim %d unsupported (must be 64)", head_dim);
    return prefill(h, stream, out, qkv, kcache, vcache, kq, vq, ks, vs, kb, vb, pos0, n_tok, n_head, n_kv_head, qkv_stride,
                   out_stride, bt, bs, "prefill_step", false, StepArgs{true, use_rope, theta});
}

extern "C" int mx230_prefill_step_proj(mx230_handle *h, void *stream, float *y, const void *w, const float *bias, int n_out,
                                       float *out, float *qkv, float *kcache, float *vcache, int8_t *kq, int8_t *vq, float *ks,
                                       float *vs, float *kb, float *vb, int pos0, int n_tok, int n_head, int n_kv_head,
                                       int head_dim, int use_rope, float theta, int qkv_stride, int out_stride, const int *bt,
                                       int bs) {
    MX_REQUIRE(head_dim == HD, MX230_ERR_UNSUPPORTED, "prefill_step_proj: head_dim %d unsupported (must be 64)", head_dim);
    MX_REQUIRE(h && y && w, MX230_ERR_INVALID_ARG, "prefill_step_proj: null argument");
    MX_REQUIRE(n_out > 0 && n_out % 8 == 0, MX230_ERR_UNSUPPORTED, "prefill_step_proj: n_out must be a multiple of 8 (got %d)", n_out);
    MX_REQUIRE((((uintptr_t)y | (uintptr_t)w | (uintptr_t)bias) & 15) == 0, MX230_ERR_INVALID_ARG,
               "prefill_step_proj: buffers must be 16-byte aligned");
    void *o_half = nullptr;
    const int rc = prefill(h, stream, out, qkv, kcache, vcache, kq, vq, ks, vs, kb, vb, pos0, n_tok, n_head, n_kv_head, qkv_stride,
                           out_stride, bt, bs, "prefill_step_proj", false, StepArgs{true, use_rope, theta}, &o_half);
    if (rc || n_tok == 0) return rc;
    mx230_device_guard guard(h->device);
    return mx230_launch_gemm_by_head(h, (cudaStream_t)stream, y, o_half, w, bias, n_tok, n_out, n_head * HD);
}
