// Batched projections either side of prefill attention: C[m][n] = A[m][k] . W[k][n] + bias[n]
// (the reference's `gemm`, 03-llm-engine/src/gpu.rs:1291-1420, called at gpu.rs:3187-3198 for qkv and
// gpu.rs:3354-3365 for the output projection; kernels gemm_f32* / gemm_half*, llm.cu).  fp32 activations in and
// out, weights fp32 or fp16 in the reference's [k][n] layout.
//
// tcgen05 with 16-bit operands and fp32 accumulation in tensor memory:
//   * fp16 weights are the B operand as they lie in memory (rows = contraction index: an MN-major operand, the
//     same descriptor form as V in the attention kernels); A is staged to fp16 once per call;
//   * fp32 weights would lose their low mantissa bits in one 16-bit operand, so both sides are staged as a
//     (high, low) pair of bf16 values, x = hi + lo to 16 bits of mantissa, and three products are accumulated:
//     A_hi W_hi + A_hi W_lo + A_lo W_hi.  The tensor cores have the time: these GEMMs are launch-bound.
// CTA = one 128 x 128 tile of C (128 x 64 where that leaves SMs idle, see mx230_gemm); k in steps of 64 through a 4-stage
// TMA ring (out-of-range rows and columns are zero-filled by the TMA unit, so m, n, k need no padding); one TMA warp, one
// MMA-issuing warp, eight epilogue warps that add the bias and hand fp32 pieces to the TMA unit.
// What bounds it at these sizes is the operands' way from L2 into shared memory (1900 x 896 x 1152: 90 MB with 64-column
// tiles, 60 MB with 128-column ones) and the launches around it.  Around the products: the bias is loaded under them, a warp's
// pieces leave through 4 KB each, staging takes two loads a thread at a time (layer of 1900 tokens, 14/2 heads, two of these
// each: 49.6 -> 47.6 us a call, 128 tokens 27.2 -> 24.6).
#include <cstring>

#include "common.cuh"

namespace {

constexpr int GM = 128, GK = 64;
constexpr int A_TILE = GM * GK * 2;   // 16 KB
constexpr int W_CHUNK = GK * 64 * 2;  // 8 KB: 64 columns (one 128-byte swizzle span) of a weight tile
constexpr int EPI_WARPS = 8;
constexpr int THREADS = (4 + EPI_WARPS) * 32;

template <bool SPLIT, int GN>
struct Smem {
    static constexpr int PARTS = SPLIT ? 2 : 1;
    static constexpr int W_TILE = GN / 64 * W_CHUNK;
    static constexpr int STAGE = PARTS * (A_TILE + W_TILE);
    static constexpr int STAGES = SPLIT && GN == 128 ? 3 : 4;   // 96 .. 192 KB
    static constexpr int BAR = STAGES * STAGE;
    static constexpr int TOTAL = BAR + 128;
    static constexpr int ALLOC = TOTAL + 1024;
};

struct GemmParams {
    float *C;
    const float *bias;
    int m, n, k;
    int a_by_head; // A is [k / 64][m][64] instead of [m][k]
    int tma_out;   // C leaves through staged TMA stores (n a multiple of 64)
    int *status;
};

// kind::f16 instruction descriptor: fp32 accumulate, A K-major, B MN-major, both operands fp16 or both bf16
__host__ __device__ constexpr uint32_t idesc(bool bf16, int GN) {
    return (1u << 4) | ((bf16 ? 1u : 0u) << 7) | ((bf16 ? 1u : 0u) << 10) | (0u << 15) | (1u << 16) |
           ((uint32_t)(GN >> 3) << 17) | ((uint32_t)(GM >> 4) << 24);
}

template <bool SPLIT, int GN>
__global__ void __launch_bounds__(THREADS, 1)
gemm_kernel(const __grid_constant__ CUtensorMap tmA0, const __grid_constant__ CUtensorMap tmA1,
            const __grid_constant__ CUtensorMap tmW0, const __grid_constant__ CUtensorMap tmW1,
            const __grid_constant__ CUtensorMap tmC, const GemmParams P) {
    using S = Smem<SPLIT, GN>;
    constexpr int STAGES = S::STAGES, W_TILE = S::W_TILE;
    extern __shared__ unsigned char smem_dyn[];
    const uint32_t smem_base = (mx::smem_u32(smem_dyn) + 1023u) & ~1023u;
    unsigned char *smem = smem_dyn + (smem_base - mx::smem_u32(smem_dyn));
    const uint32_t bar0 = smem_base + S::BAR;
    auto bar = [&](int i) { return bar0 + 8u * (uint32_t)i; };   // FULL[s] = s, EMPTY[s] = STAGES + s, ACC = 2 * STAGES
    volatile uint32_t *tmem_slot = (volatile uint32_t *)(smem + S::BAR + 8 * (2 * STAGES + 1));
    volatile int *abort_flag = (volatile int *)(smem + S::BAR + 8 * (2 * STAGES + 1) + 8);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.y * GM, n0 = blockIdx.x * GN;
    const int n_steps = (P.k + GK - 1) / GK;

    if (tid == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mx::mbar_init(bar(s), 1);
            mx::mbar_init(bar(STAGES + s), 1);
        }
        mx::mbar_init(bar(2 * STAGES), 1);
        *abort_flag = 0;
        mx::mbar_fence_init();
    }
    if (warp == 1) mx::tmem_alloc(mx::smem_u32((const void *)tmem_slot), GN);
    mx::tc_fence_before();
    __syncthreads();
    mx::tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    if (warp == 0 && lane == 0) {   // on their way into the SM's caches while the previous kernel ends
        mx::tma_prefetch_desc(&tmA0);
        mx::tma_prefetch_desc(&tmW0);
        if (SPLIT) mx::tma_prefetch_desc(&tmA1), mx::tma_prefetch_desc(&tmW1);
        if (P.tma_out) mx::tma_prefetch_desc(&tmC);
    }
    mx::pdl_wait();

    if (warp == 0) {
        // ------------------------- TMA producer -------------------------
        if (lane == 0) {
            bool ok = true;
            for (int i = 0; i < n_steps && ok; ++i) {
                const int s = i % STAGES;
                if (i >= STAGES) ok = mx::mbar_wait(bar(STAGES + s), (i / STAGES - 1) & 1, abort_flag, P.status);
                if (!ok) break;
                const uint32_t base = smem_base + s * S::STAGE;
                mx::mbar_expect_tx(bar(s), S::STAGE);
                mx::tma_load_3d(base, &tmA0, bar(s), P.a_by_head ? 0 : i * GK, m0, P.a_by_head ? i : 0);
                if (SPLIT) mx::tma_load_3d(base + A_TILE, &tmA1, bar(s), i * GK, m0, 0);
#pragma unroll
                for (int c = 0; c < GN / 64; ++c) {   // (a chunk past the last column is all zero fill)
                    mx::tma_load_3d(base + S::PARTS * A_TILE + c * W_CHUNK, &tmW0, bar(s), n0 + 64 * c, i * GK, 0);
                    if (SPLIT) mx::tma_load_3d(base + 2 * A_TILE + W_TILE + c * W_CHUNK, &tmW1, bar(s), n0 + 64 * c, i * GK, 0);
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ------------------------- MMA issuer (warp-uniform, one elected lane issues) --------------------
        constexpr uint32_t IDESC = idesc(SPLIT, GN);
        bool ok = true;
        for (int i = 0; i < n_steps && ok; ++i) {
            const int s = i % STAGES;
            ok = __all_sync(0xFFFFFFFFu, mx::mbar_wait(bar(s), (i / STAGES) & 1, abort_flag, P.status));
            if (!ok) break;
            mx::tc_fence_after();
            const uint32_t base = smem_base + s * S::STAGE;
            const uint64_t a0 = mx::smem_desc_sw128(base), w0 = mx::smem_desc_sw128_mn(base + S::PARTS * A_TILE, W_CHUNK);
            const uint64_t a1 = mx::smem_desc_sw128(base + A_TILE), w1 = mx::smem_desc_sw128_mn(base + 2 * A_TILE + W_TILE, W_CHUNK);
            if (mx::elect_one()) {
#pragma unroll
                for (int kk = 0; kk < GK / 16; ++kk) {   // A: 32 bytes per 16-element step inside the swizzle span; W: 16 rows of 128 bytes
                    mx::mma_ss(tmem, a0 + 2 * kk, w0 + 128 * kk, IDESC, (i > 0 || kk > 0));
                    if (SPLIT) {
                        mx::mma_ss(tmem, a0 + 2 * kk, w1 + 128 * kk, IDESC, 1);
                        mx::mma_ss(tmem, a1 + 2 * kk, w0 + 128 * kk, IDESC, 1);
                    }
                }
                mx::mma_commit(bar(STAGES + s));
                if (i == n_steps - 1) mx::mma_commit(bar(2 * STAGES));
            }
            __syncwarp();
        }
    } else if (warp >= 4) {
        // ------------------------- epilogue: bias, fp32 rows out -------------------------
        // warp: 32 rows (its tensor-memory lanes), half of the tile's columns
        const int q = warp & 3, colh = ((warp - 4) >> 2) * (GN / 2);
        float bias_l[GN / 64];   // lane l: the bias of column l of every piece, loaded under the products
#pragma unroll
        for (int part = 0; part < GN / 64; ++part) {
            const int col = n0 + colh + part * 32 + lane;
            bias_l[part] = P.bias && col < P.n ? P.bias[col] : 0.0f;
        }
        bool ok = __all_sync(0xFFFFFFFFu, mx::mbar_wait(bar(2 * STAGES), 0, abort_flag, P.status));
        if (ok) {
            mx::tc_fence_after();
            const int row = m0 + q * 32 + lane;
            const uint32_t ta = tmem + ((uint32_t)(q * 32) << 16);
            // pieces of 32 x 32 go through 4 KB each of the ring's first stages (every MMA has read them) and the TMA unit,
            // which clips rows past the end: 16-byte stores from lane = row registers each touch a sector of their own
            static_assert(EPI_WARPS * (GN / 64) * 4096 <= STAGES * S::STAGE, "pieces");
#pragma unroll
            for (int part = 0; part < GN / 64; ++part) {
                const int col0 = n0 + colh + part * 32;
                if (col0 >= P.n) break;
                uint32_t v[32];
                mx::tmem_ld32(ta + colh + part * 32, v);
                mx::tmem_wait_ld();
                const int st_off = ((warp - 4) * (GN / 64) + part) * 4096;
                float *crow = P.tma_out ? (float *)(smem + st_off + lane * 128) : P.C + (size_t)row * P.n + col0;
#pragma unroll
                for (int c = 0; c < 32; c += 4) {
                    float4 b4;   // (a lane past the last column has 0)
                    b4.x = __shfl_sync(0xFFFFFFFFu, bias_l[part], c), b4.y = __shfl_sync(0xFFFFFFFFu, bias_l[part], c + 1);
                    b4.z = __shfl_sync(0xFFFFFFFFu, bias_l[part], c + 2), b4.w = __shfl_sync(0xFFFFFFFFu, bias_l[part], c + 3);
                    if (col0 + c >= P.n) break;   // n is a multiple of 4: a float4 is inside or outside as a whole
                    const float4 o4 = make_float4(__uint_as_float(v[c]) + b4.x, __uint_as_float(v[c + 1]) + b4.y,
                                                  __uint_as_float(v[c + 2]) + b4.z, __uint_as_float(v[c + 3]) + b4.w);
                    if (P.tma_out) *(float4 *)((unsigned char *)crow + (((c >> 2) ^ (lane & 7)) << 4)) = o4;
                    else if (row < P.m) *(float4 *)(crow + c) = o4;
                }
                if (P.tma_out) {
                    mx::fence_proxy_async_smem();
                    __syncwarp();
                    if (lane == 0 && m0 + q * 32 < P.m) {
                        mx::tma_store_3d(&tmC, smem_base + st_off, col0 & 63, m0 + q * 32, col0 >> 6);
                        mx::bulk_commit_group();
                    }
                }
            }
            if (P.tma_out && lane == 0) mx::bulk_wait_group_read<0>();   // the pieces must outlive the reads
        }
    }
    mx::tc_fence_before();
    __syncthreads();
    mx::tc_fence_after();
    mx::pdl_trigger();   // (here, when the tensor memory is no longer wanted: the next kernel may need all of it)
    if (warp == 1) mx::tmem_dealloc(tmem, GN);
}

// Staging.  SPLIT: x -> (hi, lo) bf16 with hi = bf16(x), lo = bf16(x - hi); else x -> fp16.  Two tensors per launch
// (blockIdx.y selects): the activations, and with fp32 weights the weight matrix.
struct StageParams {
    const float *src[2];
    void *hi[2];
    void *lo[2];
    size_t n4[2];   // float4s per tensor
};

template <bool SPLIT>
__global__ void gemm_stage_kernel(StageParams P) {
    mx::pdl_trigger();
    mx::pdl_wait();
    const int t = blockIdx.y;
    const float4 *src = (const float4 *)P.src[t];
    auto convert = [&](size_t i, const float4 &x) {
        if (SPLIT) {
            const __nv_bfloat16 h0 = __float2bfloat16_rn(x.x), h1 = __float2bfloat16_rn(x.y), h2 = __float2bfloat16_rn(x.z),
                                h3 = __float2bfloat16_rn(x.w);
            const __nv_bfloat16 l0 = __float2bfloat16_rn(x.x - __bfloat162float(h0)),
                                l1 = __float2bfloat16_rn(x.y - __bfloat162float(h1)),
                                l2 = __float2bfloat16_rn(x.z - __bfloat162float(h2)),
                                l3 = __float2bfloat16_rn(x.w - __bfloat162float(h3));
            __nv_bfloat162 hv[2] = {__halves2bfloat162(h0, h1), __halves2bfloat162(h2, h3)};
            __nv_bfloat162 lv[2] = {__halves2bfloat162(l0, l1), __halves2bfloat162(l2, l3)};
            ((uint2 *)P.hi[t])[i] = *(const uint2 *)hv;
            ((uint2 *)P.lo[t])[i] = *(const uint2 *)lv;
        } else {
            __half2 hv[2] = {__floats2half2_rn(x.x, x.y), __floats2half2_rn(x.z, x.w)};
            ((uint2 *)P.hi[t])[i] = *(const uint2 *)hv;
        }
    };
    const size_t n4 = P.n4[t], step = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += 2 * step) {   // two loads in flight
        const bool two = i + step < n4;
        const float4 x = src[i], y = src[two ? i + step : i];
        convert(i, x);
        if (two) convert(i + step, y);
    }
}

// Weights of one product: fp16 as the caller has them, or a staged (high, low) pair of bf16 matrices
struct Weights {
    const void *hi, *lo;
    bool split;
};

size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

template <bool SPLIT, int GN>
int launch_tiles(mx230_handle *h, cudaStream_t st, const CUtensorMap &tA0, const CUtensorMap &tA1, const CUtensorMap &tW0,
                 const CUtensorMap &tW1, const CUtensorMap &tC, const GemmParams &P) {
    const dim3 grid((unsigned)((P.n + GN - 1) / GN), (unsigned)((P.m + GM - 1) / GM));
    MX_SMEM_ATTR_ONCE(h->device, (gemm_kernel<SPLIT, GN>), (Smem<SPLIT, GN>::ALLOC));
    MX_LAUNCH(h, st, MX230_K_GEMV, mx_launch(gemm_kernel<SPLIT, GN>, grid, THREADS, Smem<SPLIT, GN>::ALLOC, st, 1, true, tA0, tA1,
                                             tW0, tW1, tC, P));
    return MX230_OK;
}

// The GEMM itself over a staged A
int launch_gemm(mx230_handle *h, cudaStream_t st, float *C, const CUtensorMap &tA0, const CUtensorMap &tA1, bool a_by_head,
                const Weights &w, const float *bias, int m, int n, int k) {
    CUtensorMap tW0, tW1;
    const bool split = w.split;
    const int f16 = split ? 0 : 1;
    int rc = mx230_make_tmap_2d_16bit(h, &tW0, w.hi, f16, (uint64_t)n, (uint64_t)k, (uint64_t)n * 2, 64, GK);
    if (rc) return rc;
    rc = mx230_make_tmap_2d_16bit(h, &tW1, w.lo, f16, (uint64_t)n, (uint64_t)k, (uint64_t)n * 2, 64, GK);
    if (rc) return rc;

    GemmParams P;
    P.C = C, P.bias = bias, P.m = m, P.n = n, P.k = k, P.status = h->status_dev;
    P.a_by_head = a_by_head ? 1 : 0;
    // C [m][n] as [n / 64][m][64]: the store map of the attention kernels
    CUtensorMap tC;
    memset(&tC, 0, sizeof(tC));
    P.tma_out = n % 64 == 0;
    if (P.tma_out && (rc = mx230_make_tmap_f32_half_rows_strided(h, &tC, C, (uint64_t)m, (uint64_t)(n / 64), (uint64_t)n * 4, 256)))
        return rc;
    // 128-column tiles move two thirds of the bytes per CTA step that two 64-column ones do; they are taken when there are
    // enough of them for two thirds of the SMs.  (Attention half of a layer, 1900 tokens, fp16 896 x 1152 and 896 x 896: these
    // tiles, the TMA epilogue and programmatic launches of staging and GEMM 69.6 -> 55.2 us.)
    const bool wide = (long long)((n + 127) / 128) * ((m + GM - 1) / GM) * 3 >= 2ll * h->sm_count;
    if (split) rc = wide ? launch_tiles<true, 128>(h, st, tA0, tA1, tW0, tW1, tC, P) : launch_tiles<true, 64>(h, st, tA0, tA1, tW0, tW1, tC, P);
    else rc = wide ? launch_tiles<false, 128>(h, st, tA0, tA1, tW0, tW1, tC, P) : launch_tiles<false, 64>(h, st, tA0, tA1, tW0, tW1, tC, P);
    if (rc) return rc;
    MX_CHECK_CUDA(cudaGetLastError());
    return MX230_OK;
}

}  // namespace

extern "C" size_t mx230_gemm_workspace_bytes(int m, int n, int k, int weights_fp16) {
    if (m <= 0 || n <= 0 || k <= 0) return 0;
    const size_t a = align256((size_t)m * k * 2), w = align256((size_t)k * n * 2);
    return weights_fp16 ? a : 2 * a + 2 * w;
}

extern "C" int mx230_gemm(mx230_handle *h, void *stream, float *C, const float *A, const void *w, int w_fp16,
                          const float *bias, int m, int n, int k) {
    MX_REQUIRE(h && C && A && w, MX230_ERR_INVALID_ARG, "gemm: null argument");
    const float *W = w_fp16 ? nullptr : (const float *)w;
    const void *W_fp16 = w_fp16 ? w : nullptr;
    MX_REQUIRE(m >= 0 && n > 0 && k > 0, MX230_ERR_INVALID_ARG, "gemm: bad sizes %d x %d x %d", m, n, k);
    MX_REQUIRE(k % 16 == 0 && n % 8 == 0, MX230_ERR_UNSUPPORTED, "gemm: k must be a multiple of 16 and n of 8 (got k %d, n %d)", k, n);
    MX_REQUIRE((((uintptr_t)C | (uintptr_t)A | (uintptr_t)W | (uintptr_t)W_fp16 | (uintptr_t)bias) & 15) == 0,
               MX230_ERR_INVALID_ARG, "gemm: buffers must be 16-byte aligned");
    if (m == 0) return MX230_OK;
    const bool split = W != nullptr;
    const size_t need = mx230_gemm_workspace_bytes(m, n, k, split ? 0 : 1);
    MX_REQUIRE(h->ws && need <= h->ws_bytes, MX230_ERR_WORKSPACE, "gemm: workspace %zu B < %zu B needed", h->ws_bytes, need);
    h->staged.valid = 0;   // the workspace is about to hold something else
    mx230_device_guard guard(h->device);
    cudaStream_t st = (cudaStream_t)stream;
    const size_t a_bytes = align256((size_t)m * k * 2), w_bytes = align256((size_t)k * n * 2);
    unsigned char *ws = (unsigned char *)h->ws;
    void *a_hi = ws, *a_lo = ws + a_bytes, *w_hi = ws + 2 * a_bytes, *w_lo = ws + 2 * a_bytes + w_bytes;

    StageParams SP;
    SP.src[0] = A, SP.hi[0] = a_hi, SP.lo[0] = a_lo, SP.n4[0] = (size_t)m * k / 4;
    SP.src[1] = W, SP.hi[1] = w_hi, SP.lo[1] = w_lo, SP.n4[1] = split ? (size_t)k * n / 4 : 0;
    const size_t big = SP.n4[0] > SP.n4[1] ? SP.n4[0] : SP.n4[1];
    unsigned blocks = (unsigned)((big + 511) / 512);
    if (blocks > (unsigned)h->sm_count * 8) blocks = (unsigned)h->sm_count * 8;
    if (split) {
        MX_LAUNCH(h, st, MX230_K_CAST, mx_launch(gemm_stage_kernel<true>, dim3(blocks, 2), 256, 0, st, 1, true, SP));
    } else {
        MX_LAUNCH(h, st, MX230_K_CAST, mx_launch(gemm_stage_kernel<false>, dim3(blocks, 1), 256, 0, st, 1, true, SP));
    }

    CUtensorMap tA0, tA1;
    const int f16 = split ? 0 : 1;
    int rc = mx230_make_tmap_2d_16bit(h, &tA0, a_hi, f16, (uint64_t)k, (uint64_t)m, (uint64_t)k * 2, GK, GM);
    if (rc) return rc;
    rc = mx230_make_tmap_2d_16bit(h, &tA1, split ? a_lo : a_hi, f16, (uint64_t)k, (uint64_t)m, (uint64_t)k * 2, GK, GM);
    if (rc) return rc;
    return launch_gemm(h, st, C, tA0, tA1, false, split ? Weights{w_hi, w_lo, true} : Weights{W_fp16, W_fp16, false}, bias, m, n, k);
}

int mx230_launch_gemm_by_head(mx230_handle *h, cudaStream_t st, float *C, const void *A_half, const void *w, const float *bias,
                              int m, int n, int k) {
    CUtensorMap tA;   // (16-bit values and zero fill: bf16 or fp16 is the same to a copy)
    const int rc = mx230_make_tmap_bf16(h, &tA, A_half, (uint64_t)m, (uint64_t)(k / GK), GK * 2, (uint64_t)m * GK * 2, GM);
    if (rc) return rc;
    return launch_gemm(h, st, C, tA, tA, true, Weights{w, w, false}, bias, m, n, k);
}
