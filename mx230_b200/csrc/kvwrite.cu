// Per-layer attention step, part 1: RoPE and the KV-cache write (fp32 copy or int8
// quantize-on-write).  HBM-bound elementwise work; one kernel family per op, the
// reference's single / device-position / batch / per-sequence variants differ only
// in where a row's position comes from.
//
// Reference: 03-llm-engine/kernels/llm.cu:959-986 (kv_row, copy_kv_*), 1072-1117 and
// 1513-1530 (rope*), 1137-1240 and 1503-1510 (quant_affine, quantize_kv*),
// 3635-3655 (copy_kv_batch*).
#include "common.cuh"

namespace {

// Where the position of row r comes from.
//   kind 0: host scalar, row r sits at pos + r        (rope, rope_batch, *_batch)
//   kind 1: *pos_dev (one row)                        (*_dyn, graph-captured decode)
//   kind 2: pos_dev[r], block table row r of `tables` (*_seqpos, batched decode)
struct RowPos {
    int kind;
    int pos;
    const int *pos_dev;
    const int *bt;   // block table (kind 0/1) or packed tables (kind 2); null = linear
    int bs;          // block size
    int n_log;       // table row length (kind 2)
};

__device__ __forceinline__ int row_position(const RowPos &rp, int r) {
    if (rp.kind == 0) return rp.pos + r;
    if (rp.kind == 1) return *rp.pos_dev;
    return rp.pos_dev[r];
}

__device__ __forceinline__ size_t phys_row(const RowPos &rp, int r, int t) {
    const int *bt = rp.bt;
    if (bt == nullptr) return (size_t)t;
    if (rp.kind == 2) bt += (size_t)r * rp.n_log;
    return (size_t)(bt[t / rp.bs] * rp.bs + t % rp.bs);
}

// HF rotate_half RoPE, pairs (d, d + hd/2), on the Q heads then the K heads of each row.
__global__ void rope_kernel(float *qkv, RowPos rp, int n_rows, int n_head, int n_kv_head,
                            int head_dim, int stride, float theta) {
    int half = head_dim / 2;
    int per_row = (n_head + n_kv_head) * half;
    int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= n_rows * per_row) return;
    int r = idx / per_row;
    int i = idx - r * per_row;
    int h = i / half;
    int d = i - h * half;
    float *base = qkv + (size_t)r * stride + h * head_dim;
    float cs, sn;
    mx::rope_angle(row_position(rp, r), d, head_dim, theta, cs, sn);
    float x1 = base[d], x2 = base[d + half];
    mx::rope_pair(x1, x2, cs, sn);
    base[d] = x1;
    base[d + half] = x2;
}

__global__ void copy_kv_kernel(float *kcache, float *vcache, const float *qkv, RowPos rp,
                               int q_dim, int kv_dim, int stride) {
    int r = blockIdx.y;
    int i = (blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (i >= kv_dim) return;
    size_t row = phys_row(rp, r, row_position(rp, r)) * kv_dim;
    const float *src = qkv + (size_t)r * stride + q_dim;
    *(float4 *)(kcache + row + i) = *(const float4 *)(src + i);
    *(float4 *)(vcache + row + i) = *(const float4 *)(src + kv_dim + i);
}

struct SeqRows {
    float *qkv, *kcache, *vcache;
    int8_t *kq, *vq;
    float *ks, *vs, *kb, *vb;
    RowPos rp;
    int n_head, n_kv_head, stride, use_rope, max_pos;
    float theta;
};

// The work in front of a batched step's attention: a few microseconds of latency (the angle and two memory round trips), so
// what counts is that it is one launch.  It is a launch of its own because sequences may share cache blocks (several rows of
// one sequence, at consecutive positions): every row is written before any is read.  A warp takes two heads of a row,
// lane l holding dims l and l + 32, their loads issued together; the angle is formed once per warp.
// No early trigger: the attention kernel's clusters would take their places around this kernel's blocks and sit unevenly on
// the SMs (16 fp32 sequences of 1500 keys, 32/4 heads: a pass 21.9 to 25.1 us with the trigger at the top, 19.2 without).
// Against rows and attention in one launch, which cannot take rows that read one another, a batched step costs about 2 us
// more (64 int8 sequences of up to 2048 keys, 14/2 heads: 15.5 us a pass against 13.4; the case above 18.9 / 17.3); three
// separate launches took 33.3 and 32.0.
constexpr int SR_WARPS = 8, SR_UNITS = 2;
__global__ void __launch_bounds__(SR_WARPS * 32) seq_rows_kernel(const SeqRows P) {
    const int lane = threadIdx.x & 31, r = blockIdx.y;
    const float freq = P.use_rope ? mx::rope_freq(lane, 64, P.theta) : 0.0f;
    mx::pdl_wait();
    const int n_rot = P.n_head + P.n_kv_head, n_units = n_rot + P.n_kv_head;
    const int u0 = (P.use_rope ? 0 : P.n_head) + blockIdx.x * (SR_WARPS * SR_UNITS) + (threadIdx.x >> 5);
    float *row = P.qkv + (size_t)r * P.stride;
    float a[SR_UNITS], b[SR_UNITS];
#pragma unroll
    for (int i = 0; i < SR_UNITS; ++i) {
        const int u = u0 + i * SR_WARPS;
        if (u < n_units) a[i] = row[u * 64 + lane], b[i] = row[u * 64 + 32 + lane];
    }
    // (a position from device memory is kept inside the sequence's table, as in the attention kernel)
    const int pos = min(max(row_position(P.rp, r), 0), P.max_pos);
    const size_t crow = phys_row(P.rp, r, pos), kvd = (size_t)P.n_kv_head * 64;
    float cs = 1.0f, sn = 0.0f;
    if (P.use_rope && u0 < n_rot) mx::rope_angle(pos, freq, cs, sn);
#pragma unroll
    for (int i = 0; i < SR_UNITS; ++i) {
        const int u = u0 + i * SR_WARPS;
        if (u >= n_units) break;
        if (P.use_rope && u < n_rot) {
            mx::rope_pair(a[i], b[i], cs, sn);
            row[u * 64 + lane] = a[i], row[u * 64 + 32 + lane] = b[i];
        }
        if (u < P.n_head) continue;
        const bool is_v = u >= n_rot;
        const int h = is_v ? u - n_rot : u - P.n_head;
        if (P.kq == nullptr) {
            float *dst = (is_v ? P.vcache : P.kcache) + crow * kvd + h * 64;
            dst[lane] = a[i], dst[lane + 32] = b[i];
        } else {
            int8_t *dst = (is_v ? P.vq : P.kq) + crow * kvd + h * 64;
            float *be = is_v ? P.vb : P.kb;
            int c0, c1;
            float scale, beta;
            mx::quant_head_row(a[i], b[i], be != nullptr, c0, c1, scale, beta);
            dst[lane] = (int8_t)c0, dst[lane + 32] = (int8_t)c1;
            if (lane == 0) {
                (is_v ? P.vs : P.ks)[crow * P.n_kv_head + h] = scale;
                if (be != nullptr) be[crow * P.n_kv_head + h] = beta;
            }
        }
    }
}

// One warp quantises one 64-value head row (K or V) of one qkv row: lane l owns
// elements 2l, 2l+1.
__global__ void quantize_kv_kernel(int8_t *kq, int8_t *vq, float *ks, float *vs, float *kb,
                                   float *vb, const float *qkv, RowPos rp, int n_rows, int q_dim,
                                   int n_kv_head, int stride) {
    int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    int lane = threadIdx.x & 31;
    int total = n_rows * n_kv_head * 2;
    if (warp >= total) return;
    int which = warp & 1;  // 0 = K, 1 = V
    int h = (warp >> 1) % n_kv_head;
    int r = (warp >> 1) / n_kv_head;
    int kv_dim = n_kv_head * 64;
    const float *src = qkv + (size_t)r * stride + q_dim + which * kv_dim + h * 64;
    float2 x = *(const float2 *)(src + 2 * lane);
    size_t pr = phys_row(rp, r, row_position(rp, r));
    int8_t *dst = (which ? vq : kq) + pr * kv_dim + h * 64;
    float *sc = which ? vs : ks;
    float *be = which ? vb : kb;
    size_t sd = pr * n_kv_head + h;
    int c0, c1;
    float scale, beta;
    mx::quant_head_row(x.x, x.y, be != nullptr, c0, c1, scale, beta);
    if (lane == 0) {
        sc[sd] = scale;
        if (be != nullptr) be[sd] = beta;
    }
    unsigned short packed = (unsigned short)((c0 & 0xFF) | ((c1 & 0xFF) << 8));
    *(unsigned short *)(dst + 2 * lane) = packed;
}

int check_heads(const char *who, int n_head, int n_kv_head, int head_dim) {
    MX_REQUIRE(head_dim == 64, MX230_ERR_UNSUPPORTED, "%s: head_dim %d unsupported (must be 64)",
               who, head_dim);
    MX_REQUIRE(n_kv_head > 0 && n_head >= 0, MX230_ERR_INVALID_ARG, "%s: bad head counts %d/%d", who,
               n_head, n_kv_head);
    return MX230_OK;
}

int launch_rope(mx230_handle *h, void *stream, float *qkv, RowPos rp, int n_rows, int n_head,
                int n_kv_head, int head_dim, int stride, float theta) {
    MX_REQUIRE(h && qkv, MX230_ERR_INVALID_ARG, "rope: null argument");
    MX_REQUIRE(head_dim > 0 && head_dim % 2 == 0, MX230_ERR_UNSUPPORTED, "rope: odd head_dim");
    MX_REQUIRE(n_rows >= 0 && n_head >= 0 && n_kv_head >= 0, MX230_ERR_INVALID_ARG,
               "rope: negative size");
    long long total = (long long)n_rows * (n_head + n_kv_head) * (head_dim / 2);
    if (total == 0) return MX230_OK;
    mx230_device_guard guard(h->device);
    cudaStream_t st = (cudaStream_t)stream;
    MX_LAUNCH(h, st, MX230_K_ROPE, (rope_kernel<<<(unsigned)((total + 255) / 256), 256, 0, st>>>(
        qkv, rp, n_rows, n_head, n_kv_head, head_dim, stride, theta)));
    return MX230_OK;
}

int launch_copy(mx230_handle *h, void *stream, float *kcache, float *vcache, const float *qkv,
                RowPos rp, int n_rows, int q_dim, int kv_dim, int stride) {
    MX_REQUIRE(h && kcache && vcache && qkv, MX230_ERR_INVALID_ARG, "copy_kv: null argument");
    MX_REQUIRE(kv_dim > 0 && kv_dim % 4 == 0 && q_dim % 4 == 0 && stride % 4 == 0,
               MX230_ERR_UNSUPPORTED, "copy_kv: q_dim, kv_dim and stride must be multiples of 4");
    MX_REQUIRE((((uintptr_t)kcache | (uintptr_t)vcache | (uintptr_t)qkv) & 15) == 0,
               MX230_ERR_INVALID_ARG, "copy_kv: buffers must be 16-byte aligned");
    if (n_rows <= 0) return n_rows == 0 ? MX230_OK
                                        : mx230_fail(MX230_ERR_INVALID_ARG, "copy_kv: negative rows");
    mx230_device_guard guard(h->device);
    dim3 grid((kv_dim / 4 + 127) / 128, n_rows);
    cudaStream_t st = (cudaStream_t)stream;
    MX_LAUNCH(h, st, MX230_K_COPY_KV,
              (copy_kv_kernel<<<grid, 128, 0, st>>>(kcache, vcache, qkv, rp, q_dim, kv_dim, stride)));
    return MX230_OK;
}

int launch_quant(mx230_handle *h, void *stream, int8_t *kq, int8_t *vq, float *ks, float *vs,
                 float *kb, float *vb, const float *qkv, RowPos rp, int n_rows, int q_dim,
                 int n_kv_head, int head_dim, int stride) {
    MX_REQUIRE(h && kq && vq && ks && vs && qkv, MX230_ERR_INVALID_ARG,
               "quantize_kv: null argument");
    MX_REQUIRE((kb == nullptr) == (vb == nullptr), MX230_ERR_INVALID_ARG,
               "quantize_kv: kb and vb must both be given (affine) or both be null (absmax)");
    int rc = check_heads("quantize_kv", 0, n_kv_head, head_dim);
    if (rc) return rc;
    MX_REQUIRE(q_dim % 2 == 0 && stride % 2 == 0 && (((uintptr_t)qkv) & 7) == 0 &&
                   ((((uintptr_t)kq) | ((uintptr_t)vq)) & 1) == 0,
               MX230_ERR_INVALID_ARG, "quantize_kv: misaligned qkv or cache");
    if (n_rows <= 0) return n_rows == 0 ? MX230_OK
                                        : mx230_fail(MX230_ERR_INVALID_ARG, "quantize_kv: negative rows");
    mx230_device_guard guard(h->device);
    long long warps = (long long)n_rows * n_kv_head * 2;
    cudaStream_t st = (cudaStream_t)stream;
    MX_LAUNCH(h, st, MX230_K_QUANTIZE_KV,
              (quantize_kv_kernel<<<(unsigned)((warps + 3) / 4), 128, 0, st>>>(
                  kq, vq, ks, vs, kb, vb, qkv, rp, n_rows, q_dim, n_kv_head, stride)));
    return MX230_OK;
}

RowPos host_pos(int pos, const int *bt = nullptr, int bs = 0) { return RowPos{0, pos, nullptr, bt, bs, 0}; }
RowPos dev_pos(const int *p, const int *bt = nullptr, int bs = 0) { return RowPos{1, 0, p, bt, bs, 0}; }
RowPos seq_pos(const int *p, const int *tables, int bs, int n_log) {
    return RowPos{2, 0, p, tables, bs, n_log};
}

}  // namespace

int mx230_launch_seq_rows(mx230_handle *h, cudaStream_t st, float *qkv, float *kcache, float *vcache, int8_t *kq, int8_t *vq,
                          float *ks, float *vs, float *kb, float *vb, const int *pos, int n_seq, int n_head, int n_kv_head,
                          int use_rope, float theta, const int *tables, int block_size, int n_log, int qkv_stride) {
    if (kq) MX_REQUIRE(vq && ks && vs && (kb == nullptr) == (vb == nullptr), MX230_ERR_INVALID_ARG, "batched_step: missing cache array");
    else MX_REQUIRE(kcache && vcache, MX230_ERR_INVALID_ARG, "batched_step: null cache");
    MX_REQUIRE(n_head > 0 && n_kv_head > 0, MX230_ERR_INVALID_ARG, "batched_step: bad head counts %d/%d", n_head, n_kv_head);
    MX_REQUIRE(n_seq >= 0 && n_seq <= 65535, n_seq < 0 ? MX230_ERR_INVALID_ARG : MX230_ERR_UNSUPPORTED, "batched_step: n_seq %d", n_seq);
    if (n_seq == 0) return MX230_OK;
    const long long slots = (long long)block_size * n_log;
    SeqRows P{qkv, kcache, vcache, kq, vq, ks, vs, kb, vb, seq_pos(pos, tables, block_size, n_log), n_head, n_kv_head, qkv_stride,
              use_rope, (int)((slots < 0x7FFFFFFF ? slots : 0x7FFFFFFF) - 1), theta};
    mx230_device_guard guard(h->device);
    const int units = (use_rope ? n_head : 0) + 2 * n_kv_head, per = SR_WARPS * SR_UNITS;
    MX_LAUNCH(h, st, kq ? MX230_K_QUANTIZE_KV : MX230_K_COPY_KV,
              mx_launch(seq_rows_kernel, dim3((units + per - 1) / per, n_seq), SR_WARPS * 32, 0, st, 1, true, P));
    return MX230_OK;
}

// ---- rope ----
extern "C" int mx230_rope(mx230_handle *h, void *stream, float *qkv, int pos, int n_head,
                          int n_kv_head, int head_dim, float theta) {
    return launch_rope(h, stream, qkv, host_pos(pos), 1, n_head, n_kv_head, head_dim, 0, theta);
}
extern "C" int mx230_rope_dyn(mx230_handle *h, void *stream, float *qkv, const int *pos_ptr,
                              int n_head, int n_kv_head, int head_dim, float theta) {
    MX_REQUIRE(pos_ptr, MX230_ERR_INVALID_ARG, "rope_dyn: null pos_ptr");
    return launch_rope(h, stream, qkv, dev_pos(pos_ptr), 1, n_head, n_kv_head, head_dim, 0, theta);
}
extern "C" int mx230_rope_batch(mx230_handle *h, void *stream, float *qkv, int pos0, int n_tok,
                                int n_head, int n_kv_head, int head_dim, int stride, float theta) {
    return launch_rope(h, stream, qkv, host_pos(pos0), n_tok, n_head, n_kv_head, head_dim, stride,
                       theta);
}
extern "C" int mx230_rope_seqpos(mx230_handle *h, void *stream, float *qkv, const int *pos,
                                 int n_seq, int n_head, int n_kv_head, int head_dim, int stride,
                                 float theta) {
    MX_REQUIRE(pos, MX230_ERR_INVALID_ARG, "rope_seqpos: null pos");
    return launch_rope(h, stream, qkv, seq_pos(pos, nullptr, 0, 0), n_seq, n_head, n_kv_head,
                       head_dim, stride, theta);
}

// ---- fp32 KV write ----
extern "C" int mx230_copy_kv(mx230_handle *h, void *stream, float *kcache, float *vcache,
                             const float *qkv, int pos, int q_dim, int kv_dim) {
    return launch_copy(h, stream, kcache, vcache, qkv, host_pos(pos), 1, q_dim, kv_dim, 0);
}
extern "C" int mx230_copy_kv_dyn(mx230_handle *h, void *stream, float *kcache, float *vcache,
                                 const float *qkv, const int *pos_ptr, int q_dim, int kv_dim) {
    MX_REQUIRE(pos_ptr, MX230_ERR_INVALID_ARG, "copy_kv_dyn: null pos_ptr");
    return launch_copy(h, stream, kcache, vcache, qkv, dev_pos(pos_ptr), 1, q_dim, kv_dim, 0);
}
extern "C" int mx230_copy_kv_paged_dyn(mx230_handle *h, void *stream, float *kcache, float *vcache,
                                       const float *qkv, const int *pos_ptr, int q_dim, int kv_dim,
                                       const int *bt, int bs) {
    MX_REQUIRE(pos_ptr && bt && bs > 0, MX230_ERR_INVALID_ARG, "copy_kv_paged_dyn: bad table");
    return launch_copy(h, stream, kcache, vcache, qkv, dev_pos(pos_ptr, bt, bs), 1, q_dim, kv_dim, 0);
}
extern "C" int mx230_copy_kv_batch(mx230_handle *h, void *stream, float *kcache, float *vcache,
                                   const float *qkv, int pos0, int n_tok, int q_dim, int kv_dim,
                                   int stride) {
    return launch_copy(h, stream, kcache, vcache, qkv, host_pos(pos0), n_tok, q_dim, kv_dim, stride);
}
extern "C" int mx230_copy_kv_batch_paged(mx230_handle *h, void *stream, float *kcache,
                                         float *vcache, const float *qkv, int pos0, int n_tok,
                                         int q_dim, int kv_dim, int stride, const int *bt, int bs) {
    MX_REQUIRE(bt && bs > 0, MX230_ERR_INVALID_ARG, "copy_kv_batch_paged: bad table");
    return launch_copy(h, stream, kcache, vcache, qkv, host_pos(pos0, bt, bs), n_tok, q_dim, kv_dim,
                       stride);
}
extern "C" int mx230_copy_kv_seqpos(mx230_handle *h, void *stream, float *kcache, float *vcache,
                                    const float *qkv, const int *pos, int n_seq, int q_dim,
                                    int kv_dim, int qkv_stride, const int *tables, int block_size,
                                    int n_log) {
    MX_REQUIRE(pos && tables && block_size > 0, MX230_ERR_INVALID_ARG, "copy_kv_seqpos: bad table");
    return launch_copy(h, stream, kcache, vcache, qkv, seq_pos(pos, tables, block_size, n_log), n_seq,
                       q_dim, kv_dim, qkv_stride);
}

// ---- int8 quantize-on-write ----
extern "C" int mx230_quantize_kv(mx230_handle *h, void *stream, int8_t *kq, int8_t *vq, float *ks,
                                 float *vs, float *kb, float *vb, const float *qkv, int pos,
                                 int q_dim, int n_kv_head, int head_dim) {
    return launch_quant(h, stream, kq, vq, ks, vs, kb, vb, qkv, host_pos(pos), 1, q_dim, n_kv_head,
                        head_dim, 0);
}
extern "C" int mx230_quantize_kv_dyn(mx230_handle *h, void *stream, int8_t *kq, int8_t *vq,
                                     float *ks, float *vs, float *kb, float *vb, const float *qkv,
                                     const int *pos_ptr, int q_dim, int n_kv_head, int head_dim) {
    MX_REQUIRE(pos_ptr, MX230_ERR_INVALID_ARG, "quantize_kv_dyn: null pos_ptr");
    return launch_quant(h, stream, kq, vq, ks, vs, kb, vb, qkv, dev_pos(pos_ptr), 1, q_dim,
                        n_kv_head, head_dim, 0);
}
extern "C" int mx230_quantize_kv_paged_dyn(mx230_handle *h, void *stream, int8_t *kq, int8_t *vq,
                                           float *ks, float *vs, float *kb, float *vb,
                                           const float *qkv, const int *pos_ptr, int q_dim,
                                           int n_kv_head, int head_dim, const int *bt, int bs) {
    MX_REQUIRE(pos_ptr && bt && bs > 0, MX230_ERR_INVALID_ARG, "quantize_kv_paged_dyn: bad table");
    return launch_quant(h, stream, kq, vq, ks, vs, kb, vb, qkv, dev_pos(pos_ptr, bt, bs), 1, q_dim,
                        n_kv_head, head_dim, 0);
}
extern "C" int mx230_quantize_kv_batch(mx230_handle *h, void *stream, int8_t *kq, int8_t *vq,
                                       float *ks, float *vs, float *kb, float *vb,
                                       const float *qkv, int pos0, int n_tok, int q_dim,
                                       int n_kv_head, int head_dim, int stride) {
    return launch_quant(h, stream, kq, vq, ks, vs, kb, vb, qkv, host_pos(pos0), n_tok, q_dim,
                        n_kv_head, head_dim, stride);
}
extern "C" int mx230_quantize_kv_batch_paged(mx230_handle *h, void *stream, int8_t *kq, int8_t *vq,
                                             float *ks, float *vs, float *kb, float *vb,
                                             const float *qkv, int pos0, int n_tok, int q_dim,
                                             int n_kv_head, int head_dim, int stride,
                                             const int *bt, int bs) {
    MX_REQUIRE(bt && bs > 0, MX230_ERR_INVALID_ARG, "quantize_kv_batch_paged: bad table");
    return launch_quant(h, stream, kq, vq, ks, vs, kb, vb, qkv, host_pos(pos0, bt, bs), n_tok, q_dim,
                        n_kv_head, head_dim, stride);
}
extern "C" int mx230_quantize_kv_seqpos(mx230_handle *h, void *stream, int8_t *kq, int8_t *vq,
                                        float *ks, float *vs, float *kb, float *vb,
                                        const float *qkv, const int *pos, int n_seq, int q_dim,
                                        int n_kv_head, int head_dim, int qkv_stride,
                                        const int *tables, int block_size, int n_log) {
    MX_REQUIRE(pos && tables && block_size > 0, MX230_ERR_INVALID_ARG,
               "quantize_kv_seqpos: bad table");
    return launch_quant(h, stream, kq, vq, ks, vs, kb, vb, qkv,
                        seq_pos(pos, tables, block_size, n_log), n_seq, q_dim, n_kv_head, head_dim,
                        qkv_stride);
}
