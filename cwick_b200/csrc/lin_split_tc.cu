// lin_split_tc.cu -- y[t] = W x[t] for a chunk of tokens with f32 activations and bf16 weights, on the tensor cores
// without giving up the activations' precision: the projections, the absorb and the un-absorb of the reference-named
// chunk entry point (cwick_linear's BF16 branch, src/tensor.c:143-176; src/attention.c:741-744, :812-815; batched over the
// chunk's tokens as src/attention.c:943-1024 does).
//
// An f32 activation is written as the sum of three bf16 numbers (its rounding, the rounding of what is left, and again),
// which is the f32 value to the last bit or nearly; a product with a bf16 weight is then three bf16 products, accumulated
// in f32 in tensor memory like everything else. Three MMAs per product at 1.6 PFLOP/s against CUDA-core f32 multiply-adds:
// the four projections of a 512-token chunk of a 4096-wide layer took 2.84 ms on CUDA cores and take 0.13 ms here.
//
// One block = one tile of 128 tokens x BN outputs x one part of the contraction. Bound: per 64-wide step three planes of
// 16 KB and 32 KB of weights arrive (80 KB) for 12 MMAs of 128 cycles; an SM takes some 56 B/clk from L2, so loads (1.43 k
// cycles) and MMAs (1.54 k) are in balance, which is why the tile is 256 outputs wide: at 128 the loads alone would be
// 1.17 k cycles for 0.77 k of MMAs. Weights come from HBM once per token tile and have a ring of their own, four steps
// deep; the planes come from L2 and have two. A tile that would leave SMs idle has its contraction split, the partial
// sums added by the kernel that reads them next (a norm, the split into planes, the sum).
// Padding (a chunk's last tile, or one of a few tokens) costs no more than the weights' own time: 12 x 128 cycles per 32 KB
// of weights are 19 us for 109 MB of them on 148 SMs, and HBM needs 17 us.
//
// Every mbarrier wait is bounded and records a code in the context's error word when it gives up.
#include <algorithm>

#include "lin_split_tc.cuh"
#include "tc_common.cuh"

namespace {

constexpr int LS_TOK = 128, LS_BK = 64;
constexpr int LS_PLANE = LS_TOK * LS_BK * 2;              // 16384
template <int P, int BN>
struct LsCfg {
    static constexpr int A_BYTES = P * LS_PLANE, W_BYTES = BN * LS_BK * 2;
    static constexpr int NA = P == 1 ? 4 : 2, NW = 4;
    static constexpr int OFF_A = 0, OFF_W = NA * A_BYTES, OFF_BAR = OFF_W + NW * W_BYTES;
    static constexpr int SMEM = OFF_BAR + 256 + 1024;
    static_assert(SMEM <= 232448, "shared-memory budget");
    static_assert(NW * W_BYTES >= 8 * 4096, "the epilogue's staging tiles lie in the weight ring");
};

struct LsParams {
    int n, k, rows, rows2, nb1, heads, splits;
    int64_t w_head_rows, w_row_off, ldy;
    void *y;
    int *err;
};

__device__ __forceinline__ void split3(float x, uint16_t &a, uint16_t &b, uint16_t &c) {
    const __nv_bfloat16 h = __float2bfloat16_rn(x);
    const float r1 = x - __bfloat162float(h);
    const __nv_bfloat16 m = __float2bfloat16_rn(r1);
    const __nv_bfloat16 l = __float2bfloat16_rn(r1 - __bfloat162float(m));
    a = __bfloat16_as_ushort(h); b = __bfloat16_as_ushort(m); c = __bfloat16_as_ushort(l);
}
// two neighbours at once, packed as they lie in memory
__device__ __forceinline__ void split3x2(float x, float y, uint32_t (&o)[3]) {
    uint16_t a0, b0, c0, a1, b1, c1;
    split3(x, a0, b0, c0);
    split3(y, a1, b1, c1);
    o[0] = a0 | ((uint32_t)a1 << 16); o[1] = b0 | ((uint32_t)b1 << 16); o[2] = c0 | ((uint32_t)c1 << 16);
}

// P planes of A; BN outputs per tile; WK: W's rows are the contraction index; OUT as CwkSplitGemm::Out.
// grid (output tiles, token tiles, heads or splits), 256 threads: warp 0 loads, warp 1 issues the MMAs, all eight write out.
template <int P, int BN, bool WK, int OUT>
__global__ void __launch_bounds__(256, 1)
lin_split_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_w2,
                 const LsParams p) {
    using C = LsCfg<P, BN>;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t *sm = smem_raw + (base - raw);
    const uint32_t bar0 = base + C::OFF_BAR;
    enum { AF = 0, AE = 4, WF = 8, WE = 12, DONE = 16, NBAR = 17 };
    auto bar = [&](int i) { return bar0 + 8u * (uint32_t)i; };
    uint32_t *s_tmem = reinterpret_cast<uint32_t *>(sm + C::OFF_BAR + 8 * NBAR + 8);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const bool second = (int)blockIdx.x >= p.nb1;
    const int c0 = ((int)blockIdx.x - (second ? p.nb1 : 0)) * BN;         // first output of the tile, within its matrix
    const int t0 = (int)blockIdx.y * LS_TOK;
    const int head = p.heads > 1 ? (int)blockIdx.z : 0, part = p.heads > 1 ? 0 : (int)blockIdx.z;
    const int nkb = p.k / LS_BK;
    const int kb0 = (int)((int64_t)nkb * part / p.splits), kb1 = (int)((int64_t)nkb * (part + 1) / p.splits);

    if (tid == 0) {
        asm volatile("prefetch.tensormap [%0];" ::"l"(&tm_a) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(second ? &tm_w2 : &tm_w) : "memory");
        for (int i = 0; i < NBAR; i++) mbar_init(bar(i), 1u);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    cwk_pdl_launch();
    cwk_pdl_wait();
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(s_tmem)), "r"((uint32_t)BN) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *s_tmem;

    if (warp == 0 && lane == 0) {
        const CUtensorMap *tw = second ? &tm_w2 : &tm_w;
        bool ok = true;
        int wi = 0, ai = 0;                                // copies issued
        for (int i = 0; kb0 + i < kb1 && ok; i++) {
            const int kb = kb0 + i;
            const int ws = i % C::NW, as = i % C::NA;
            ok = mbar_wait(bar(WE + ws), (uint32_t)(((i / C::NW) & 1) ^ 1), p.err, 1201);
            if (!ok) break;
            mbar_expect_tx(bar(WF + ws), C::W_BYTES);
            if (WK) tma_load_3d(base + C::OFF_W + ws * C::W_BYTES, tw, 0, (int)(head * p.w_head_rows + p.w_row_off) + kb * LS_BK, c0 / 64, bar(WF + ws));
            else tma_load_3d(base + C::OFF_W + ws * C::W_BYTES, tw, 0, (int)(head * p.w_head_rows + p.w_row_off) + c0, kb, bar(WF + ws));
            wi = i + 1;
            ok = mbar_wait(bar(AE + as), (uint32_t)(((i / C::NA) & 1) ^ 1), p.err, 1202);
            if (!ok) break;
            mbar_expect_tx(bar(AF + as), C::A_BYTES);
            tma_load_4d(base + C::OFF_A + as * C::A_BYTES, &tm_a, 0, t0, head * nkb + kb, 0, bar(AF + as));
            ai = i + 1;
        }
        if (!ok) {                                         // the copies still in flight
            for (int j = (wi > C::NW ? wi - C::NW : 0); j < wi; j++) mbar_wait(bar(WF + j % C::NW), (uint32_t)((j / C::NW) & 1), p.err, 1203);
            for (int j = (ai > C::NA ? ai - C::NA : 0); j < ai; j++) mbar_wait(bar(AF + j % C::NA), (uint32_t)((j / C::NA) & 1), p.err, 1204);
        }
    } else if (warp == 1 && lane == 0) {
        constexpr uint32_t ID = idesc_bf16(128, BN, 0, WK ? 1 : 0);
        bool ok = true;
        for (int i = 0; kb0 + i < kb1 && ok; i++) {
            const int ws = i % C::NW, as = i % C::NA;
            ok = mbar_wait(bar(WF + ws), (uint32_t)((i / C::NW) & 1), p.err, 1205);
            if (ok) ok = mbar_wait(bar(AF + as), (uint32_t)((i / C::NA) & 1), p.err, 1206);
            if (!ok) break;
            tc_fence_after();
            const uint64_t dA = smem_desc(base + C::OFF_A + as * C::A_BYTES, 16, 1024);
            const uint64_t dW = WK ? smem_desc(base + C::OFF_W + ws * C::W_BYTES, LS_BK * 128, 1024) : smem_desc(base + C::OFF_W + ws * C::W_BYTES, 16, 1024);
#pragma unroll
            for (int pl = 0; pl < P; pl++)
#pragma unroll
                for (int s = 0; s < 4; s++)
                    umma_bf16(tmem, dA + (uint64_t)((pl * LS_PLANE + s * 32) >> 4), dW + (uint64_t)((s * (WK ? 2048 : 32)) >> 4), ID,
                              (uint32_t)((i | pl | s) != 0));
            umma_commit(bar(WE + ws));
            umma_commit(bar(AE + as));
        }
        if (ok) umma_commit(bar(DONE));
    }
    __syncwarp();
    // ---- epilogue: a thread holds one token row of 32 lanes' worth; 128-byte lines leave through a per-warp staging tile,
    // which lies in the weight ring (every copy into it has been consumed once DONE is complete)
    if (mbar_wait_warp(bar(DONE), 0, p.err, 1207)) {
        tc_fence_after();
        const int q4 = warp & 3, g2 = warp >> 2;
        const uint32_t tlane = tmem + ((uint32_t)(q4 * 32) << 16);
        uint8_t *stg = sm + C::OFF_W + warp * 4096;
        const int t0w = t0 + q4 * 32;
        const int lim = second ? p.rows2 : p.rows;         // outputs of this matrix
        const int64_t ybase = (int64_t)head * p.rows + (second ? p.rows : 0);
        auto put = [&](const uint32_t (&w)[32]) {          // this thread's 128 bytes of the staging tile
#pragma unroll
            for (int j = 0; j < 8; j++)
                *reinterpret_cast<uint4 *>(stg + lane * 128 + ((j ^ (lane & 7)) << 4)) = make_uint4(w[4 * j], w[4 * j + 1], w[4 * j + 2], w[4 * j + 3]);
            __syncwarp();
        };
        auto flush = [&](uint8_t *y0, int64_t row_bytes, int el, int col) {      // lines of row t0w + .. at column `col`
#pragma unroll
            for (int r8 = 0; r8 < 8; r8++) {
                const int rr = r8 * 4 + (lane >> 3), jj = lane & 7;
                const uint4 w = *reinterpret_cast<const uint4 *>(stg + rr * 128 + ((jj ^ (rr & 7)) << 4));
                if (t0w + rr < p.n && col + (jj + 1) * (16 / el) <= lim)
                    *reinterpret_cast<uint4 *>(y0 + (int64_t)(t0w + rr) * row_bytes + (ybase + col) * el + jj * 16) = w;
            }
            __syncwarp();
        };
#pragma unroll 1
        for (int c = 0; c < BN / 128; c++) {
            const int col = (g2 * (BN / 128) + c) * 64;
            if (c0 + col >= lim) break;
            uint32_t v[64];
            TMEM_LD16(v, 0, tlane + col);
            TMEM_LD16(v, 16, tlane + col + 16);
            TMEM_LD16(v, 32, tlane + col + 32);
            TMEM_LD16(v, 48, tlane + col + 48);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            uint32_t w[32];
            if (OUT == CwkSplitGemm::F32) {
                uint8_t *y0 = (uint8_t *)p.y + (int64_t)part * p.n * p.ldy * 4;
#pragma unroll
                for (int u = 0; u < 2; u++) {
#pragma unroll
                    for (int j = 0; j < 32; j++) w[j] = v[u * 32 + j];
                    put(w);
                    flush(y0, p.ldy * 4, 4, c0 + col + u * 32);
                }
            } else if (OUT == CwkSplitGemm::BF16) {
#pragma unroll
                for (int j = 0; j < 32; j++) w[j] = pack_bf16x2(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1]));
                put(w);
                flush((uint8_t *)p.y, p.ldy * 2, 2, c0 + col);
            } else {
#pragma unroll 1
                for (int pl = 0; pl < CWK_PLANES; pl++) {
#pragma unroll
                    for (int j = 0; j < 32; j++) {         // (the remainders go back into v: the next plane splits what is left)
                        const float x = __uint_as_float(v[2 * j]), y = __uint_as_float(v[2 * j + 1]);
                        w[j] = pack_bf16x2(x, y);
                        v[2 * j] = __float_as_uint(x - __uint_as_float(w[j] << 16));
                        v[2 * j + 1] = __float_as_uint(y - __uint_as_float(w[j] & 0xffff0000u));
                    }
                    put(w);
                    flush((uint8_t *)p.y + (int64_t)pl * p.n * p.ldy * 2, p.ldy * 2, 2, c0 + col);
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)BN) : "memory");
    }
}

__global__ void __launch_bounds__(256) split_planes_kernel(const float4 *x, int64_t quads, uint2 *o) {
    const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
    cwk_pdl_launch();
    cwk_pdl_wait();
    if (i >= quads) return;
    const float4 v = x[i];
    uint32_t a[3], b[3];
    split3x2(v.x, v.y, a);
    split3x2(v.z, v.w, b);
#pragma unroll
    for (int pl = 0; pl < 3; pl++) o[pl * quads + i] = make_uint2(a[pl], b[pl]);
}

__global__ void __launch_bounds__(256) sum_partials_kernel(const float4 *part, int splits, int64_t quads, float4 *out, uint2 *planes) {
    const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
    cwk_pdl_launch();
    cwk_pdl_wait();
    if (i >= quads) return;
    float4 v = part[i];
    for (int s = 1; s < splits; s++) {
        const float4 w = part[s * quads + i];
        v.x += w.x; v.y += w.y; v.z += w.z; v.w += w.w;
    }
    if (out) out[i] = v;
    if (planes) {
        uint32_t a[3], b[3];
        split3x2(v.x, v.y, a);
        split3x2(v.z, v.w, b);
#pragma unroll
        for (int pl = 0; pl < 3; pl++) planes[pl * quads + i] = make_uint2(a[pl], b[pl]);
    }
}

bool encode(CUtensorMap *tm, const void *ptr, int rank, const cuuint64_t *dims, const cuuint64_t *strides, const cuuint32_t *box) {
    const cuuint32_t es[4] = {1, 1, 1, 1};
    return cwk_encode_tiled_fn()(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rank, const_cast<void *>(ptr), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                 CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int P, int BN, bool WK, int OUT>
int launch(cwk_ctx *ctx, const CwkSplitGemm &g) {
    using C = LsCfg<P, BN>;
    CUtensorMap ta, tw, tw2;
    {
        // A as [64][tokens][k blocks][planes]: a step is one box of 128 tokens x one block x every plane
        const cuuint64_t dims[4] = {64, (cuuint64_t)g.n, (cuuint64_t)(g.lda / 64), (cuuint64_t)P};
        const cuuint64_t strides[3] = {(cuuint64_t)g.lda * 2, 128, (cuuint64_t)g.n * g.lda * 2};
        const cuuint32_t box[4] = {64, LS_TOK, 1, P};
        if (!encode(&ta, g.A, 4, dims, strides, box)) return cwk_fail(ctx, CWK_ERR_CUDA, "cuTensorMapEncodeTiled failed for a projection's activations");
    }
    for (int i = 0; i < 2; i++) {
        // W as [64][rows][column blocks]: a step is BN rows x one block, or (WK) 64 rows x BN / 64 blocks
        const bool two = i == 1 && g.W2;
        const cuuint64_t dims[3] = {64, (cuuint64_t)(two ? g.rows2 : g.w_rows), (cuuint64_t)(g.ldw / 64)};
        const cuuint64_t strides[2] = {(cuuint64_t)g.ldw * 2, 128};
        const cuuint32_t box[3] = {64, WK ? (cuuint32_t)LS_BK : (cuuint32_t)BN, WK ? (cuuint32_t)(BN / 64) : 1u};
        if (!encode(i ? &tw2 : &tw, two ? g.W2 : g.W, 3, dims, strides, box)) return cwk_fail(ctx, CWK_ERR_CUDA, "cuTensorMapEncodeTiled failed for a projection's weights");
    }
    static bool attr_set[16] = {false};
    if (!attr_set[ctx->device & 15]) {
        CWK_CUDA(ctx, cudaFuncSetAttribute(lin_split_kernel<P, BN, WK, OUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM));
        attr_set[ctx->device & 15] = true;
    }
    LsParams p;
    p.n = g.n; p.k = g.k; p.rows = g.rows; p.rows2 = g.W2 ? g.rows2 : 0; p.heads = g.heads; p.splits = g.splits;
    p.nb1 = (g.rows + BN - 1) / BN;
    p.w_head_rows = g.w_head_rows; p.w_row_off = g.w_row_off; p.ldy = g.ldy; p.y = g.Y; p.err = ctx->dev_err;
    const dim3 grid((unsigned)(p.nb1 + (g.W2 ? (g.rows2 + BN - 1) / BN : 0)), (unsigned)((g.n + LS_TOK - 1) / LS_TOK),
                    (unsigned)(g.heads > 1 ? g.heads : g.splits));
    CWK_CUDA(ctx, cwk_launch_early(lin_split_kernel<P, BN, WK, OUT>, grid, dim3(256), C::SMEM, ctx->stream, ta, tw, tw2, p));
    CWK_LAUNCH_CHECK(ctx, "lin_split_kernel");
    return CWK_OK;
}

}  // namespace

bool cwk_split_gemm_ok(const CwkSplitGemm &g) {
    if (!cwk_encode_tiled_fn()) return false;
    if (g.k % 64 || g.lda % 64 || g.ldw % 64 || g.rows % 8 || g.rows2 % 8 || g.ldy % 8 || g.n <= 0 || g.k <= 0) return false;
    return ((reinterpret_cast<uintptr_t>(g.A) | reinterpret_cast<uintptr_t>(g.W) | reinterpret_cast<uintptr_t>(g.W2) | reinterpret_cast<uintptr_t>(g.Y)) & 15) == 0;
}

// One wave of blocks: as many parts as there are SMs for the tiles, each at least four steps long.
int cwk_split_gemm_splits(const cwk_ctx *ctx, int n, int rows, int rows2, int k) {
    const int tiles = ((rows + 255) / 256 + (rows2 + 255) / 256) * ((n + LS_TOK - 1) / LS_TOK);
    return std::max(1, std::min(ctx->sm_count / std::max(1, tiles), k / LS_BK / 4));
}

int cwk_split_gemm(cwk_ctx *ctx, const CwkSplitGemm &g) {
    int s = cwk_ensure_err_word(ctx);
    if (s != CWK_OK) return s;
    if (g.planes == 3 && !g.w_k_rows && g.out == CwkSplitGemm::F32) return launch<3, 256, false, CwkSplitGemm::F32>(ctx, g);
    if (g.planes == 3 && !g.w_k_rows && g.out == CwkSplitGemm::PLANES) return launch<3, 256, false, CwkSplitGemm::PLANES>(ctx, g);
    if (g.planes == 3 && g.w_k_rows && g.out == CwkSplitGemm::BF16) return launch<3, 256, true, CwkSplitGemm::BF16>(ctx, g);
    if (g.planes == 1 && !g.w_k_rows && g.out == CwkSplitGemm::PLANES) return launch<1, 128, false, CwkSplitGemm::PLANES>(ctx, g);
    return cwk_fail(ctx, CWK_ERR_UNSUPPORTED, "lin_split: combination not built");
}

int cwk_split_planes(cwk_ctx *ctx, const float *x, int n, int k, uint16_t *planes) {
    const int64_t quads = (int64_t)n * k / 4;
    CWK_CUDA(ctx, cwk_launch_early(split_planes_kernel, dim3((unsigned)((quads + 255) / 256)), dim3(256), 0, ctx->stream, (const float4 *)x, quads, (uint2 *)planes));
    CWK_LAUNCH_CHECK(ctx, "split_planes_kernel");
    return CWK_OK;
}

int cwk_sum_partials(cwk_ctx *ctx, const float *part, int splits, int n, int cols, float *out, uint16_t *planes) {
    const int64_t quads = (int64_t)n * cols / 4;
    CWK_CUDA(ctx, cwk_launch_early(sum_partials_kernel, dim3((unsigned)((quads + 255) / 256)), dim3(256), 0, ctx->stream, (const float4 *)part, splits, quads, (float4 *)out, (uint2 *)planes));
    CWK_LAUNCH_CHECK(ctx, "sum_partials_kernel");
    return CWK_OK;
}
