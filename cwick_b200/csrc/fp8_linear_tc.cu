// fp8_linear_tc.cu -- the FP8-E4M3 block-scaled projection on tcgen05.
//
//   Y[n][cols] = sum over 128-wide K blocks kb of  scale[col/128][kb] * ( X[:, kb] . W[:, kb]^T )
//
// The E4M3 codes are first widened to bf16 by a small kernel (exact: every E4M3
// value is a bf16 value), so the contraction is a bf16 x bf16 MMA with exact
// products and f32 accumulation. The F32 block scale changes every 128 along K
// and is not representable in the operands without rounding, so each K block is
// accumulated on its own in tensor memory and then multiplied by its scale and
// added into f32 registers by the epilogue warps ("block sum times scale", the
// order of src/tensor.c:511-520). Two TMEM accumulators alternate so the MMA of
// block kb+1 runs while block kb is being promoted.
//
// A pair of CTAs (a cluster of two) takes tiles of 256 rows of X x 256 outputs (two scale column blocks), K step 128 = one
// scale block per pipeline stage, three stages. The tile's MMA spans the pair (M 256 x N 256): each CTA holds its own 128
// rows of X and one half of the 256 weight rows, so that 64 KB per SM and step arrive for 1024 cycles of MMAs. With a
// 128 x 256 tile per SM it was 96 KB, and the ~56 B/clk an SM gets from L2 while all of them load made the step 1.8 k cycles
// (o_proj, 4096 tokens, 8192 -> 4096: 251 us). An operand tile arrives as ONE TMA box of two 64-wide column blocks (a TMA
// operation costs some 400 cycles whatever its size).
// The pairs are persistent: whole waves of tiles first; the tiles left over are cut along K into parts so that the last
// round is as full as the others (a chunk of a few tiles is all last round), their partial sums added by a second kernel.
// Warp 0 = TMA producer, warp 1 = TMEM owner and, in the pair's first CTA, MMA issuer for both, warps 4..11 = promotion /
// epilogue of the CTA's own 128 rows (TMEM lane quarter = warp % 4; warps 4-7 own output columns 0-127 of the tile,
// warps 8-11 columns 128-255); they write out while the next tile's first blocks are multiplied. The issuing warp runs its loop
// as a whole with one lane elected for the MMAs, and the promotion works on pairs of columns: 4096 tokens on their own 202 -> 178 us
// (o_proj), 138 -> 128 (q_b), 64 -> 58 (q_a and kv_a). A whole prompt of that size is at the power cap and gains nothing from it.
#include <algorithm>
#include <map>
#include <tuple>

#include "tc_common.cuh"

namespace {

constexpr int BM = CWK_FP8_TILE, BN = CWK_FP8_TILE, BK = 128;
constexpr int STAGES = 3;
constexpr int A_BYTES = BM / 2 * BK * 2, B_BYTES = BN / 2 * BK * 2;   // 32 KB + 32 KB per CTA
constexpr int G_OFF_STG = STAGES * (A_BYTES + B_BYTES);          // 196608: eight 4 KB staging tiles of the epilogue
constexpr int G_OFF_BAR = G_OFF_STG + 8 * 4096;
constexpr int G_SMEM = G_OFF_BAR + 256 + 1024;
constexpr uint32_t G_TMEM_COLS = 512;                             // two 256-column partial accumulators
constexpr int G_THREADS = 384;
enum { GB_FULL = 0, GB_EMPTY = STAGES, GB_PFULL = 2 * STAGES, GB_PEMPTY = 2 * STAGES + 2, GB_COUNT = 2 * STAGES + 4 };

// E4M3 -> bf16, exact. 16 codes per thread.
__global__ void __launch_bounds__(256) e4m3_to_bf16_kernel(const uint8_t *src, uint16_t *dst, int64_t n16) {
    const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (i >= n16) return;
    const uint4 v = reinterpret_cast<const uint4 *>(src)[i];
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    uint32_t o[8];
#pragma unroll
    for (int k = 0; k < 4; k++)
#pragma unroll
        for (int hlf = 0; hlf < 2; hlf++) {
            uint32_t r = 0;
#pragma unroll
            for (int j = 0; j < 2; j++) {
                const uint32_t b = (w[k] >> (16 * hlf + 8 * j)) & 0xffu;
                const uint32_t e = (b >> 3) & 15u, m = b & 7u;
                uint32_t h;
                if (e == 0) {
                    if (m == 0) h = 0;
                    else {
                        const int lz = (m >= 4) ? 0 : (m >= 2 ? 1 : 2);
                        h = ((uint32_t)(120 - lz) << 7) | (((m << (lz + 1)) & 7u) << 4);
                    }
                } else if (e == 15 && m == 7) h = 0x7fc0u;
                else h = ((e + 120u) << 7) | (m << 4);
                h |= (b & 0x80u) << 8;
                r |= h << (16 * j);
            }
            o[k * 2 + hlf] = r;
        }
    reinterpret_cast<uint4 *>(dst)[2 * i] = make_uint4(o[0], o[1], o[2], o[3]);
    reinterpret_cast<uint4 *>(dst)[2 * i + 1] = make_uint4(o[4], o[5], o[6], o[7]);
}

// One launch serves one projection, or two that share the activations X (q_a and kv_a of the MLA
// prefill): column tiles [0, tiles_a) belong to the first weight matrix, the rest to the second.
struct GemmProblem {
    const float *scale_inv;
    int64_t cols;
    void *Y;
    int out_bf16;
};
struct GemmParams {
    GemmProblem pr[2];
    int tiles_a, tiles_n, tiles_m;   // column tiles of the first problem and of both, row tiles
    int full, splits;                // tiles done whole; parts of K each later tile is cut into
    float *part;                     // partial sums of the cut tiles [tile - full][part][256][256]
    int64_t n, k;
    int *err;
};

struct GemmUnit {
    int second, col0, row0, kb0, kb1, slot;      // slot: which partial-sum tile (-1: a whole tile)
};
// Work unit u: tiles 0 .. full - 1, then the parts of the tiles after them. Row tiles vary fastest: pairs that run at the
// same time share weight tiles and, between them, all of X.
__device__ __forceinline__ GemmUnit gemm_unit(int u, const GemmParams &p, int nkb) {
    GemmUnit g;
    int tile = u, part = 0, parts = 1;
    g.slot = -1;
    if (u >= p.full && p.splits > 1) {
        tile = p.full + (u - p.full) / p.splits;
        part = (u - p.full) % p.splits;
        parts = p.splits;
        g.slot = u - p.full;
    }
    const int tn = tile / p.tiles_m;
    g.second = tn >= p.tiles_a;
    g.col0 = (tn - (g.second ? p.tiles_a : 0)) * BN;
    g.row0 = (tile % p.tiles_m) * BM;
    g.kb0 = nkb * part / parts;
    g.kb1 = nkb * (part + 1) / parts;
    return g;
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(G_THREADS, 1)
fp8_linear_tc_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_w,
                     const __grid_constant__ CUtensorMap tm_w2, const GemmParams p) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t *sm = smem_raw + (base - raw);
    const uint32_t bar0 = base + G_OFF_BAR;
    auto bar = [&](int i) { return bar0 + 8u * (uint32_t)i; };
    uint32_t *s_tmem = reinterpret_cast<uint32_t *>(sm + G_OFF_BAR + 8 * GB_COUNT + 8);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rank = (int)cluster_rank();
    const int nkb = (int)(p.k / 128);              // scale blocks along K = pipeline steps
    const int units = p.splits > 1 ? p.full + (p.tiles_n * p.tiles_m - p.full) * p.splits : p.tiles_n * p.tiles_m;
    const int u0 = (int)blockIdx.x >> 1, du = (int)gridDim.x >> 1;

    if (tid == 0) {
        asm volatile("prefetch.tensormap [%0];" ::"l"(&tm_x) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&tm_w) : "memory");
        if (p.tiles_n > p.tiles_a) asm volatile("prefetch.tensormap [%0];" ::"l"(&tm_w2) : "memory");
        for (int i = 0; i < GB_COUNT; i++) mbar_init(bar(i), (i >= GB_PEMPTY) ? 16u : 1u);      // PEMPTY: the promotion warps of both CTAs
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    cwk_pdl_launch();
    cwk_pdl_wait();
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(s_tmem)), "r"(G_TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();
    tc_fence_after();
    const uint32_t tmem = *s_tmem;

    if (warp == 0) {
        if (lane == 0) {
            bool ok = true;
            int c = 0;                                       // steps issued so far, over all units
            for (int u = u0; u < units && ok; u += du) {
                const GemmUnit g = gemm_unit(u, p, nkb);
                for (int kb = g.kb0; kb < g.kb1 && ok; kb++, c++) {
                    const int slot = c % STAGES, use = c / STAGES;
                    ok = mbar_wait(bar(GB_EMPTY + slot), (uint32_t)((use & 1) ^ 1), p.err, 401);
                    if (!ok) break;
                    // both CTAs' tiles are counted at the first CTA's barrier, where the issuer waits
                    if (rank == 0) mbar_expect_tx(bar(GB_FULL + slot), 2 * (A_BYTES + B_BYTES));
                    const uint32_t full = cluster_addr(bar(GB_FULL + slot), 0), a0 = base + slot * (A_BYTES + B_BYTES);
                    tma_load_3d_pair(a0, &tm_x, 0, g.row0 + rank * (BM / 2), kb * 2, full);
                    // (the maps are kernel parameters: their addresses must stay in parameter space, so no pointer select)
                    if (g.second) tma_load_3d_pair(a0 + A_BYTES, &tm_w2, 0, g.col0 + rank * (BN / 2), kb * 2, full);
                    else tma_load_3d_pair(a0 + A_BYTES, &tm_w, 0, g.col0 + rank * (BN / 2), kb * 2, full);
                }
            }
            // the issuer commits to both CTAs: none of these arrivals may still be on its way here when this CTA leaves
            for (int s = max(0, c - STAGES); s < c && ok; s++)
                ok = mbar_wait(bar(GB_EMPTY + s % STAGES), (uint32_t)((s / STAGES) & 1), p.err, 406);
            if (!ok && rank == 0)      // drain the copies still in flight before leaving
                for (int s = (c > STAGES ? c - STAGES : 0); s < c; s++)
                    mbar_wait(bar(GB_FULL + s % STAGES), (uint32_t)((s / STAGES) & 1), p.err, 402);
        }
    } else if (warp == 1) {
        if (rank == 0) {
            uint32_t patience = WAIT_LIMIT;
            constexpr uint32_t ID = idesc_bf16(BM, BN, 0, 0);
            const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
            const uint64_t da0 = smem_desc(base, 16, 1024), db0 = smem_desc(base + A_BYTES, 16, 1024);
            int c = 0, slot = 0, use = 0;
            for (int u = u0; u < units; u += du) {
                const GemmUnit g = gemm_unit(u, p, nkb);
#pragma unroll 1
                for (int kb = g.kb0; kb < g.kb1; kb++, c++) {
                    const int pb = c & 1, puse = c >> 1;
                    mbar_wait_on(bar(GB_FULL + slot), (uint32_t)(use & 1), p.err, 404, patience);
                    mbar_wait_on(bar(GB_PEMPTY + pb), (uint32_t)((puse & 1) ^ 1), p.err, 403, patience);
                    tc_fence_after();
                    const uint64_t off = (uint64_t)((slot * (A_BYTES + B_BYTES)) >> 4);
                    if (elect_one()) {
#pragma unroll
                        for (int ks = 0; ks < 8; ks++)          // 64-wide column block ks >> 2 of each operand, 32 bytes per 16-wide step
                            umma_bf16_pair(tm + pb * 256, da0 + off + (uint64_t)(((ks >> 2) * (BM / 2 * 128) + (ks & 3) * 32) >> 4),
                                           db0 + off + (uint64_t)(((ks >> 2) * (BN / 2 * 128) + (ks & 3) * 32) >> 4), ID, ks != 0);
                        umma_commit_pair(bar(GB_PFULL + pb));
                        umma_commit_pair(bar(GB_EMPTY + slot));        // stage may be refilled once these MMAs are done
                    }
                    __syncwarp();
                    if (++slot == STAGES) { slot = 0; use++; }
                }
            }
            settle(patience != WAIT_LIMIT);
        }
    } else if (warp >= 4) {
        const int q = warp & 3, ch = (warp - 4) >> 2;
        const uint32_t tlane = tmem + ((uint32_t)(q * 32) << 16);
        const int64_t ncb = (p.k + 127) / 128;
        uint8_t *stg = sm + G_OFF_STG + (warp - 4) * 4096;
        bool ok = true;
        int c = 0;
        for (int u = u0; u < units && ok; u += du) {
            const GemmUnit g = gemm_unit(u, p, nkb);
            // (field-wise selects: indexing the parameter struct with a run-time index would copy it to local memory)
            const int64_t cols = g.second ? p.pr[1].cols : p.pr[0].cols;
            const int cbase = g.col0 + ch * 128;             // first output column of this warp's 128
            const bool live = cbase < cols;                  // a tile past the last column block: only keep the barriers moving
            const float *srow = (g.second ? p.pr[1].scale_inv : p.pr[0].scale_inv) + (int64_t)(live ? cbase / 128 : 0) * ncb;
            uint64_t acc2[64];                               // f32 pairs: promoted two at a time
#pragma unroll
            for (int j = 0; j < 64; j++) acc2[j] = 0;
            for (int kb = g.kb0; kb < g.kb1; kb++, c++) {
                const int pb = c & 1, puse = c >> 1;
                ok = mbar_wait_warp(bar(GB_PFULL + pb), (uint32_t)(puse & 1), p.err, 405);
                if (!ok) break;
                tc_fence_after();
                if (live) {
                    const float sc = __ldg(srow + kb);
                    const uint64_t sc2 = ((uint64_t)__float_as_uint(sc) << 32) | __float_as_uint(sc);
#pragma unroll
                    for (int cc = 0; cc < 4; cc++) {
                        uint32_t v[32];                              // two loads in flight per wait
                        TMEM_LD16(v, 0, tlane + pb * 256 + ch * 128 + cc * 32);
                        TMEM_LD16(v, 16, tlane + pb * 256 + ch * 128 + cc * 32 + 16);
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                        for (int j = 0; j < 16; j++) {
                            const uint64_t x = ((uint64_t)v[2 * j + 1] << 32) | v[2 * j];
                            asm("fma.rn.ftz.f32x2 %0, %1, %2, %0;" : "+l"(acc2[cc * 16 + j]) : "l"(x), "l"(sc2));
                        }
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster(cluster_addr(bar(GB_PEMPTY + pb), 0));
            }
            if (!ok || !live) continue;
            float acc[128];
#pragma unroll
            for (int j = 0; j < 64; j++) {
                acc[2 * j] = __uint_as_float((uint32_t)acc2[j]);
                acc[2 * j + 1] = __uint_as_float((uint32_t)(acc2[j] >> 32));
            }
            // A thread holds one row; whole 128-byte lines leave through the warp's staging tile, four rows per instruction.
            const int r0 = g.row0 + rank * (BM / 2) + q * 32;
            const bool bf16 = g.slot < 0 && (g.second ? p.pr[1].out_bf16 : p.pr[0].out_bf16);
            uint8_t *y;                                          // row r0, column cbase
            int64_t row_bytes;
            int rows_left, cols_left = (int)(cols - cbase);
            if (g.slot >= 0) {
                row_bytes = BN * 4;
                y = (uint8_t *)(p.part + (int64_t)g.slot * BM * BN + (int64_t)(rank * (BM / 2) + q * 32) * BN + ch * 128);
                rows_left = 32; cols_left = 128;
            } else {
                row_bytes = cols * (bf16 ? 2 : 4);
                y = (uint8_t *)(g.second ? p.pr[1].Y : p.pr[0].Y) + (int64_t)r0 * row_bytes + (int64_t)cbase * (bf16 ? 2 : 4);
                rows_left = (int)min((int64_t)32, p.n - r0);
            }
            auto flush = [&](int col, int el) {                  // the staging tile's 128 bytes per row, at column `col` (8-column pieces are whole)
                __syncwarp();
#pragma unroll
                for (int r8 = 0; r8 < 8; r8++) {
                    const int rr = r8 * 4 + (lane >> 3), jj = lane & 7;
                    const uint4 w = *reinterpret_cast<const uint4 *>(stg + rr * 128 + ((jj ^ (rr & 7)) << 4));
                    if (rr < rows_left && col + (jj + 1) * (16 / el) <= cols_left) *reinterpret_cast<uint4 *>(y + (int64_t)rr * row_bytes + col * el + jj * 16) = w;
                }
                __syncwarp();
            };
            if (bf16) {
#pragma unroll
                for (int cc = 0; cc < 2; cc++) {
#pragma unroll
                    for (int j = 0; j < 8; j++)
                        *reinterpret_cast<uint4 *>(stg + lane * 128 + ((j ^ (lane & 7)) << 4)) =
                            make_uint4(pack_bf16x2(acc[cc * 64 + 8 * j], acc[cc * 64 + 8 * j + 1]), pack_bf16x2(acc[cc * 64 + 8 * j + 2], acc[cc * 64 + 8 * j + 3]),
                                       pack_bf16x2(acc[cc * 64 + 8 * j + 4], acc[cc * 64 + 8 * j + 5]), pack_bf16x2(acc[cc * 64 + 8 * j + 6], acc[cc * 64 + 8 * j + 7]));
                    flush(cc * 64, 2);
                }
            } else {
#pragma unroll
                for (int cc = 0; cc < 4; cc++) {
#pragma unroll
                    for (int j = 0; j < 8; j++)
                        *reinterpret_cast<float4 *>(stg + lane * 128 + ((j ^ (lane & 7)) << 4)) =
                            make_float4(acc[cc * 32 + 4 * j], acc[cc * 32 + 4 * j + 1], acc[cc * 32 + 4 * j + 2], acc[cc * 32 + 4 * j + 3]);
                    flush(cc * 32, 4);
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();                                          // the pair's barriers and tensor memory stay until both are done
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(G_TMEM_COLS) : "memory");
    }
}

// Adds up the parts of the tiles that were cut along K, in order. Four columns per thread, 64 threads per row.
__global__ void __launch_bounds__(256) fp8_sum_parts_kernel(const GemmParams p) {
    cwk_pdl_launch();
    cwk_pdl_wait();
    const int tile = p.full + (int)blockIdx.y, tn = tile / p.tiles_m;
    const bool second = tn >= p.tiles_a;
    const int row = (int)blockIdx.x * 4 + (int)(threadIdx.x >> 6), c = (int)(threadIdx.x & 63) * 4;
    const int64_t r = (int64_t)(tile % p.tiles_m) * BM + row, col = (int64_t)(tn - (second ? p.tiles_a : 0)) * BN + c;
    const int64_t cols = second ? p.pr[1].cols : p.pr[0].cols;
    if (r >= p.n || col >= cols) return;                     // (cols is a multiple of 8: four columns are in or out together)
    const float *src = p.part + (int64_t)blockIdx.y * p.splits * BM * BN + row * BN + c;
    float4 v = *reinterpret_cast<const float4 *>(src);
#pragma unroll 4
    for (int s = 1; s < p.splits; s++) {
        const float4 w = *reinterpret_cast<const float4 *>(src + (int64_t)s * BM * BN);
        v.x += w.x; v.y += w.y; v.z += w.z; v.w += w.w;
    }
    void *Y = second ? p.pr[1].Y : p.pr[0].Y;
    if (second ? p.pr[1].out_bf16 : p.pr[0].out_bf16)
        *reinterpret_cast<uint2 *>((uint16_t *)Y + r * cols + col) = make_uint2(pack_bf16x2(v.x, v.y), pack_bf16x2(v.z, v.w));
    else
        *reinterpret_cast<float4 *>((float *)Y + r * cols + col) = v;
}

}  // namespace

bool cwk_fp8_linear_tc_available() { return true; }

// Widened copies of weight tensors, kept per context. A serving loop applies the same few projections to every
// chunk, and checkpoints are immutable (the reference maps them read-only), so the exact E4M3 -> bf16 widening of a
// weight is done once per (pointer, shape) and reused, up to a byte budget; beyond it, or after
// cwk_ctx_drop_weight_cache, a call widens into the context's transient buffer as before.
struct WideEntry {
    void *dev;
    CUtensorMap tm;
};
struct WideCache {
    std::map<std::tuple<const void *, int64_t, int64_t>, WideEntry> m;
    size_t bytes = 0;
};

void cwk_fp8_weight_cache_free(cwk_ctx *ctx) {
    WideCache *wc = (WideCache *)ctx->wide_cache;
    if (!wc) return;
    for (auto &kv : wc->m) cudaFree(kv.second.dev);
    delete wc;
    ctx->wide_cache = nullptr;
}

static int encode_weight_map(cwk_ctx *ctx, const void *dst, int64_t cols, int64_t k, CUtensorMap *tm);

// Widens W (E4M3 [cols][k]) to bf16 and encodes its tensor map: from the context's cache when the weight has been
// seen, into the cache when it has room, else into the context's transient buffer at element offset `at`.
static int prepare_weights(cwk_ctx *ctx, const void *W, int64_t cols, int64_t k, size_t at, CUtensorMap *tm) {
    const int64_t n16 = cols * k / 16;
    const size_t bytes = (size_t)cols * k * 2;
    if (!ctx->wide_cache) ctx->wide_cache = new WideCache();
    WideCache *wc = (WideCache *)ctx->wide_cache;
    const auto key = std::make_tuple(W, cols, k);
    auto it = wc->m.find(key);
    if (it != wc->m.end()) { *tm = it->second.tm; return CWK_OK; }
    uint16_t *dst = (uint16_t *)ctx->wbf16 + at;
    bool cached = false;
    if (wc->bytes + bytes <= ctx->wide_cache_budget) {
        void *d = nullptr;
        if (cudaMalloc(&d, bytes) == cudaSuccess) { dst = (uint16_t *)d; cached = true; }
        else (void)cudaGetLastError();
    }
    e4m3_to_bf16_kernel<<<(unsigned)((n16 + 255) / 256), 256, 0, ctx->stream>>>((const uint8_t *)W, dst, n16);
    CWK_LAUNCH_CHECK(ctx, "e4m3_to_bf16_kernel");
    int s = encode_weight_map(ctx, dst, cols, k, tm);
    if (s != CWK_OK) { if (cached) cudaFree(dst); return s; }
    if (cached) {
        wc->m[key] = WideEntry{dst, *tm};
        wc->bytes += bytes;
    }
    return CWK_OK;
}

static int encode_weight_map(cwk_ctx *ctx, const void *dst_c, int64_t cols, int64_t k, CUtensorMap *tm) {
    void *dst = const_cast<void *>(dst_c);
    CwkEncodeTiledFn enc = cwk_encode_tiled_fn();
    cuuint32_t es[3] = {1, 1, 1};
    cuuint64_t wd[3] = {64, (cuuint64_t)cols, (cuuint64_t)(k / 64)};
    cuuint64_t st[2] = {(cuuint64_t)k * 2, 128};
    cuuint32_t wb[3] = {64, BN / 2, 2};
    if (enc(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, dst, wd, st, wb, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return cwk_fail(ctx, CWK_ERR_CUDA, "cuTensorMapEncodeTiled failed for the projection weights");
    return CWK_OK;
}

// Y1 = X . W1^T (block-scaled), and, when W2 is given, Y2 = X . W2^T in the same launch. left: where the parts of the tiles that were
// cut along K are, for a caller whose next kernel adds them up itself (NULL: added up here). They stay until the stream's next launch after that kernel.
int cwk_fp8_linear_tc_launch2(cwk_ctx *ctx, const void *X, int64_t n, int64_t k, const void *W1, const float *scale1, int64_t cols1,
                              void *Y1, int out_bf16_1, const void *W2, const float *scale2, int64_t cols2, void *Y2, int out_bf16_2, CwkFp8Parts *left) {
    // vector stores in the epilogue want 16-byte aligned rows
    if ((cols1 % 8) != 0 || (k % 128) != 0 || ((uintptr_t)Y1 % 16) != 0 || ((uintptr_t)X % 16) != 0 ||
        (W2 && ((cols2 % 8) != 0 || ((uintptr_t)Y2 % 16) != 0)))
        return cwk_fail(ctx, CWK_ERR_UNSUPPORTED, "tcgen05 FP8 GEMM needs cols %% 8 == 0 and k %% 128 == 0");
    if (!cwk_encode_tiled_fn()) return cwk_fail(ctx, CWK_ERR_UNSUPPORTED, "cuTensorMapEncodeTiled not available");
    {
        int es = cwk_ensure_err_word(ctx);
        if (es != CWK_OK) return es;
    }
    // widened weights live in their own buffer (the split scratch and the prefill workspace are in use around this call)
    const size_t e1 = (size_t)cols1 * k, e2 = W2 ? (size_t)cols2 * k : 0;
    const size_t wbytes = (e1 + e2) * 2;
    if (wbytes > ctx->wbf16_bytes) {
        if (ctx->wbf16) {
            CWK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
            CWK_CUDA(ctx, cudaFree(ctx->wbf16));
            ctx->wbf16 = nullptr;
            ctx->wbf16_bytes = 0;
        }
        CWK_CUDA(ctx, cudaMalloc(&ctx->wbf16, wbytes));
        ctx->wbf16_bytes = wbytes;
    }
    CUtensorMap tm_x, tm_w, tm_w2;
    int s = prepare_weights(ctx, W1, cols1, k, 0, &tm_w);
    if (s != CWK_OK) return s;
    tm_w2 = tm_w;
    if (W2) {
        s = prepare_weights(ctx, W2, cols2, k, e1, &tm_w2);
        if (s != CWK_OK) return s;
    }
    {
        // activations as [64][rows][k / 64 column blocks]: one box = all rows of a tile x two column blocks (one 128-wide scale block)
        CwkEncodeTiledFn enc = cwk_encode_tiled_fn();
        cuuint32_t es[3] = {1, 1, 1};
        cuuint64_t xd[3] = {64, (cuuint64_t)n, (cuuint64_t)(k / 64)};
        cuuint64_t st[2] = {(cuuint64_t)k * 2, 128};
        cuuint32_t xb[3] = {64, BM / 2, 2};
        if (enc(&tm_x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void *>(X), xd, st, xb, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return cwk_fail(ctx, CWK_ERR_CUDA, "cuTensorMapEncodeTiled failed for the projection activations");
    }
    static bool attr_set[16] = {false};
    if (!attr_set[ctx->device & 15]) {
        CWK_CUDA(ctx, cudaFuncSetAttribute(fp8_linear_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, G_SMEM));
        attr_set[ctx->device & 15] = true;
    }
    GemmParams p;
    p.pr[0].scale_inv = scale1; p.pr[0].cols = cols1; p.pr[0].Y = Y1; p.pr[0].out_bf16 = out_bf16_1;
    p.pr[1] = p.pr[0];
    if (W2) { p.pr[1].scale_inv = scale2; p.pr[1].cols = cols2; p.pr[1].Y = Y2; p.pr[1].out_bf16 = out_bf16_2; }
    p.tiles_a = (int)((cols1 + BN - 1) / BN);
    p.tiles_n = p.tiles_a + (W2 ? (int)((cols2 + BN - 1) / BN) : 0);
    p.tiles_m = (int)((n + BM - 1) / BM);
    p.n = n; p.k = k; p.err = ctx->dev_err;
    // Whole waves, then the rest cut along K into as many parts as fill one more round, each at least four blocks long.
    const int pairs = std::max(1, ctx->sm_count / 2), tiles = p.tiles_n * p.tiles_m;
    p.full = tiles / pairs * pairs;
    const int rest = tiles - p.full;
    p.splits = rest > 0 ? std::max(1, std::min(pairs / rest, (int)(k / 128 / 4))) : 1;
    p.part = nullptr;
    if (p.splits > 1) {
        s = cwk_reserve_scratch(ctx, (size_t)rest * p.splits * BM * BN * 4);
        if (s != CWK_OK) return s;
        p.part = ctx->scratch;
    }
    const int units = p.full + rest * p.splits;
    CwkKernelTimer timer(ctx);
    CWK_CUDA(ctx, cwk_launch_early(fp8_linear_tc_kernel, dim3(2 * std::min(units, pairs)), dim3(G_THREADS), G_SMEM, ctx->stream, tm_x, tm_w, tm_w2, p));
    CWK_LAUNCH_CHECK(ctx, "fp8_linear_tc_kernel");
    if (left) *left = CwkFp8Parts{p.part, p.full, p.splits, p.tiles_m, p.tiles_a};
    else if (p.splits > 1) {
        CWK_CUDA(ctx, cwk_launch_early(fp8_sum_parts_kernel, dim3(BM / 4, (unsigned)rest), dim3(256), 0, ctx->stream, p));
        CWK_LAUNCH_CHECK(ctx, "fp8_sum_parts_kernel");
    }
    return CWK_OK;
}

int cwk_fp8_linear_tc_launch(cwk_ctx *ctx, const void *X, const void *W, const float *scale_inv, int64_t n, int64_t k,
                             int64_t cols, void *Y, int out_bf16) {
    return cwk_fp8_linear_tc_launch2(ctx, X, n, k, W, scale_inv, cols, Y, out_bf16, nullptr, nullptr, 0, nullptr, 0, nullptr);
}
