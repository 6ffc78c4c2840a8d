// mla_prefill_attn.cu -- causal MLA prefill attention with the queries as the MMA's rows.
//
// The decode kernel (mla_decode_tc.cu) treats a query token as 64 rows (its heads) of a 576-wide
// product against the latent cache; run once per token of a prompt, its MMAs are 64 columns wide,
// bound by shared-memory bandwidth, and every 128-key tile is a serial chain. A prompt has a better
// shape: per HEAD, 128 consecutive tokens are the 128 rows of an MMA. Scores are taken against the
// head's expanded key, not against the latent:
//
//   s[t][h][c] = q_nope[t][h] . (W_uk[h] lat[c])  +  q_rope[t][h] . k_rope[c]        (192-wide)
//   out[t][h]  = sum_c softmax_c(s) lat[c]                                            (512-wide)
//
// which is the absorbed attention of src/attention.c:741-782 with the product W_uk^T q_nope . lat
// re-associated: the same scores, 192 instead of 576 multiply-adds each, and the values are still the
// shared latent, so the output is the absorbed [tokens][heads][512] result. Two kernels:
//
//   kexp_tc_kernel: Kx[h][c][0:128] = W_uk[h] lat[c] (tcgen05, W_uk[h] resident per block as the
//     K-major B operand, latent tiles streamed), Kx[h][c][128:192] = k_rope[c]. Head-major: a head's 64-key tile is
//     24 KB of consecutive memory (token-major rows would lie 24 KB apart and crowd a few L2 slices).
//   The attention: one item = 128 queries x one head. The accumulator of one half of the 512 value columns, 128 x 256 f32, is half of
//     tensor memory, so an item is two blocks' work. Keys stream in tiles of 64 (24 KB), latent halves beside them (32 KB), one TMA box
//     each. The query tile sits in tensor memory (96 columns of bf16 pairs) as the A operand of the score MMAs, which
//     so read only the keys from shared memory.
//     Per tile: S = Q Kx^T (12 MMAs, M 128 x N 64) into one of two TMEM score buffers; the softmax
//     warps own one query row per thread (TMEM lane = row, so row maxima and sums need no shuffles),
//     write P (bf16); O += P lat (4 MMAs, M 128 x N 256). The two products have
//     issuers of their own, so the scores run ahead of the values and the tensor pipe works under the softmax.
//     There are two forms. The fast one (prefill_pair_kernel; GQA: prefill_attn_kernel<4>) splits the 64 keys of a row between two
//     softmax warp groups (two threads per row, another two groups for every other tile) and never rescales: a row's reference
//     exponent is its largest score of the first tile, later scores may outrun it by up to 2^64 (bf16 P and the f32 accumulators have
//     the range), and a block that sees more raises a flag. The exact one (prefill_attn_kernel<1>: one thread per row, each half
//     for itself, lazy rescale of its own TMEM lane when a score outruns the reference by 2^8) runs right after it and recomputes the
//     flagged items only.
//
// Every mbarrier wait is bounded and records a code in the context's error word when it gives up.
#include <algorithm>

#include "tc_common.cuh"

namespace {

constexpr int PA_QT = 128, PA_KT = 64, PA_DV = 256, PA_L = 512, PA_ROW = 576;
constexpr int PA_C_BYTES = PA_KT * PA_DV * 2;         // 32768: four [64][64] blocks
constexpr int PA_P_BYTES = PA_QT * PA_KT * 2;         // 16384: one [128][64] block
constexpr int PA_KST = 3;
// "Key tile here" has more barriers than the ring has slots: tile kc arrives at barrier kc % PA_KBAR. The two score issuers take
// alternate tiles, so with one barrier per slot an issuer would wait for every SECOND phase of it, and a parity wait cannot tell
// that phase from the one two before: with the copy of tile kc - 3 late and that of kc - 2 not, the issuer of kc - 2 went
// on to kc before its slot had been filled. With an even number of barriers each has one issuer, which sees all of its phases.
constexpr int PA_KBAR = 2 * PA_KST;
constexpr int PA_OFF_K = 0;                            // (the query tile lives in tensor memory, not here)
// prefill_attn_kernel serves two shapes. MLA prefill (its exact form): 192-wide expanded keys, the 512 value columns in two halves, three
// value stages. GQA prefill (Qwen3.5 layers): 256-wide keys and values of one KV head, two value stages (the key tiles are
// 32 KB instead of 24 KB). Shared-memory layout and the query tile's width in tensor memory follow from DQK and CST.
template <int DQK_, int CST_>
struct PaCfg {
    static constexpr int DQK = DQK_, CST = CST_;
    static constexpr int K_BYTES = PA_KT * DQK * 2;    // 24576 / 32768: DQK / 64 blocks of [64][64]
    static constexpr int OFF_C = PA_OFF_K + PA_KST * K_BYTES;
    static constexpr int OFF_P = OFF_C + CST * PA_C_BYTES;
    static constexpr int OFF_BAR = OFF_P + 2 * PA_P_BYTES;
    static constexpr int OFF_X = OFF_BAR + 512;        // [4][128] f32 maxima, [4][128] f32 sums exchanged between the softmax groups; 8 items of 16 bytes
    static constexpr int SMEM = OFF_X + 4096 + 128 + 1024;
    static_assert(SMEM <= 232448, "shared-memory budget");
    static_assert(384 + DQK / 2 <= 512, "tensor-memory budget");
};
using PaMla = PaCfg<192, 3>;
using PaGqa = PaCfg<256, 2>;
static_assert(PaMla::OFF_BAR == 204800, "shared-memory budget");
constexpr uint32_t PA_COL_O = 0, PA_COL_S = 256, PA_COL_Q = 384;   // S buffers at 256 and 320; Q: DQK / 2 columns of bf16 pairs
constexpr float PA_LAZY = 8.f;                         // exact form: rescale when a score outruns the reference by 2^8
constexpr float PA_RANGE = 64.f;                       // fast form: flag the block when a score outruns it by 2^64
constexpr int PA_SBUF = 2;                             // score buffers in tensor memory
enum { PB_QFULL = 0, PB_KFULL = 1, PB_KEMPTY = PB_KFULL + PA_KBAR, PB_CFULL = PB_KEMPTY + PA_KST, PB_CEMPTY = PB_CFULL + 3, PB_SFULL = PB_CEMPTY + 3,
       PB_SEMPTY = PB_SFULL + 2, PB_PFULL = PB_SEMPTY + 2, PB_PEMPTY = PB_PFULL + 2, PB_ODONE = PB_PEMPTY + 2, PB_QEMPTY, PB_OFREE, PB_XM, PB_XL, PB_ITEM,
       PB_COUNT = PB_ITEM + 8 };
static_assert(PA_KBAR % 2 == 0 && PA_KBAR % PA_KST == 0 && 8 * PB_COUNT + 16 <= 512, "barriers");

struct AttnParams {
    const uint16_t *q;  // bf16 [n][nh][DQK]
    const float4 *rot;  // MLA: [n][32] (cos, sin) of the rope pairs, two pairs a piece; NULL: q is rotated already
    uint16_t *out;      // bf16 [n][nh][512] (MLA) / [n][nh][256] (GQA)
    int n, nh, T;       // T = pos0 + n cached rows
    int group;          // GQA: query heads per KV head (MLA: unused)
    int64_t pos0;
    float scale_log2;
    int *flags;         // one word per item (share mode: per item + share): fast form sets it, exact form runs only where it is set
    int *counter;       // [3]: item counters of the fast and the exact form, number of flags raised; zero at launch
    int *err;
    // Share mode (shares > 0): the key tiles of all items, one after another, are dealt out to the blocks (MLA: pairs of blocks) in
    // equal contiguous shares, whatever the items' number and lengths; what a share has of an item that is not all its own is left
    // as a record (record_of), and attn_merge_kernel joins them.
    int shares;         // number of blocks or pairs
    int head_tiles;     // key tiles of one head
    float *records;     // [2 * shares] (MLA: times two halves) [PA_RECORD]
};
constexpr int PA_RECORD = PA_QT * (PA_DV + 2);         // floats: O as [PA_DV / 4][row][4], m [row], l [row]

struct AttnItem {
    int q0, h, half, lo, nt;   // key tiles lo .. nt - 1
    int rec, flag;             // where the result goes as a record (-1: into the output); index of the flag
};

// Work item w of the attention grid: query tiles from the longest to the shortest inside one head, then the next head: blocks that
// run at the same time work on the same few heads, whose keys stay in L2. (MLA: each of the two halves of the value columns does it.)
__device__ __forceinline__ AttnItem attn_item(int w, const AttnParams &p, int nq) {
    AttnItem it;
    const int qtile = nq - 1 - (w % nq);
    it.q0 = qtile * PA_QT;
    it.h = w / nq;
    it.half = 0;
    const int64_t last_q = p.pos0 + min(it.q0 + PA_QT - 1, p.n - 1);     // keys 0 .. pos0 + (last query of the item): tiles of 64
    it.lo = 0;
    it.nt = (int)(last_q / PA_KT) + 1;
    it.rec = -1;
    it.flag = w;
    return it;
}

// Share mode: where an item is cut. A segment's first tile must show every row of the item a key (the rows' reference
// exponents come from it): cuts inside the diagonal move down to its first tile.
__device__ __forceinline__ int attn_cut(int tile, const AttnItem &it, const AttnParams &p) {
    return tile <= 0 ? 0 : tile >= it.nt ? it.nt : min(tile, (int)((p.pos0 + it.q0) / PA_KT));
}
// total_tiles * g / shares, in 32 bits (the launch sees to it that there are less than 2^31 tiles)
__device__ __forceinline__ int64_t share_begin(int g, int64_t total_tiles, int shares) {
    const uint32_t t = (uint32_t)total_tiles, q = t / (uint32_t)shares, r = t - q * (uint32_t)shares;
    return (int64_t)(q * (uint32_t)g + r * (uint32_t)g / (uint32_t)shares);
}
template <bool GQA> __device__ __forceinline__ int64_t record_of(int rec, int half) { return GQA ? rec : 2 * rec + half; }
// The part of share g (tiles u0 .. u1 - 1 of all) in item `it`, which begins at tile `at` of all; false: none.
__device__ __forceinline__ bool attn_segment(AttnItem &it, int w, int g, int64_t at, int64_t u0, int64_t u1, const AttnParams &p) {
    const int nt = it.nt, lo = attn_cut((int)max((int64_t)-1, min((int64_t)nt, u0 - at)), it, p), hi = attn_cut((int)max((int64_t)-1, min((int64_t)nt, u1 - at)), it, p);
    it.lo = lo;
    it.nt = hi;
    it.rec = lo > 0 ? 2 * g : hi < nt ? 2 * g + 1 : -1;      // (only a share's first segment begins inside an item, only its last ends inside one)
    it.flag = w + g;                                         // (from one segment to the next w or g goes up)
    return hi > lo;
}

// Two f32 in one register pair and the arithmetic on both at once (half the instructions of the softmax: its warps, not the
// tensor pipe, are what a tile waits for).
__device__ __forceinline__ uint64_t pack_f32x2(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack_f32x2(uint64_t v, float &a, float &b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint64_t add_f32x2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// The query tile is the A operand of every score MMA of the item; it is kept in tensor memory (row = lane, two
// consecutive bf16 per 32-bit column), so that those MMAs read only the keys from shared memory. A thread
// copies its row's share: DQK / 2 columns split between the groups. The tile of item k + 1 is copied
// BEFORE the epilogue of item k, so that the next item's first scores are computed under that epilogue.
template <class CFG, int NWG, bool GQA, class F>      // NWG copying groups; done: says so for the warp
__device__ __forceinline__ void load_query_tile(const AttnParams &p, int q0_, int h_, int row, int wg, uint32_t tlane, F done) {
    const int t = q0_ + row;
    const uint4 *src = reinterpret_cast<const uint4 *>(p.q + ((int64_t)t * p.nh + h_) * CFG::DQK);
#pragma unroll
    for (int c = 0; c < CFG::DQK / 16 / NWG; c++) {        // eight words at a time, the groups in turn
        const int w8 = c * NWG + wg;
        uint32_t wv[8];
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const uint4 v = (t < p.n) ? src[w8 * 2 + j] : make_uint4(0, 0, 0, 0);
            wv[4 * j] = v.x; wv[4 * j + 1] = v.y; wv[4 * j + 2] = v.z; wv[4 * j + 3] = v.w;
        }
        // the rope pairs (the last 64 of 192 columns) are rotated on their way, at the row's position: a kernel of its own, in
        // place, was 32 us for 4096 tokens of 64 heads, 13 for 509
        if (!GQA && c * NWG * 16 >= CFG::DQK - 64 && p.rot && t < p.n) {
#pragma unroll
            for (int j = 0; j < 8; j += 2) {
                const float4 r = p.rot[(int64_t)t * 16 + w8 * 4 - (CFG::DQK - 64) / 4 + j / 2];
                const float a0 = __uint_as_float(wv[j] << 16), b0 = __uint_as_float(wv[j] & 0xffff0000u);
                const float a1 = __uint_as_float(wv[j + 1] << 16), b1 = __uint_as_float(wv[j + 1] & 0xffff0000u);
                wv[j] = pack_bf16x2(a0 * r.x - b0 * r.y, b0 * r.x + a0 * r.y);
                wv[j + 1] = pack_bf16x2(a1 * r.z - b1 * r.w, b1 * r.z + a1 * r.w);
            }
        }
        TMEM_ST8(wv, 0, tlane + PA_COL_Q + w8 * 8);
    }
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    tc_fence_before();
    done();
}

// Softmax groups and tiles. A tile's scores go from tensor memory through registers into P in a chain (barrier, load, maximum,
// exponentials, barrier, store, fence) that takes longer than its MMAs. So in the fast form two of the four groups take the even tiles
// and two the odd ones, a row's 64 keys between them, and the chains of two tiles overlap.
//
// Persistent: one block per SM takes items from a global counter until none is left. The first TMA operation of a
// block waits several thousand cycles for its tensor map, tensor memory is allocated once, and the loads of the next
// item run under the epilogue of this one.
template <int NWG> constexpr int PA_THREADS = 128 + 128 * NWG + (NWG == 4 ? 32 : 0);      // (the last warp: second issuer of the scores)
template <int NWG, class CFG, bool GQA>      // NWG softmax warp groups: 4 = fast form, 1 = exact form
__global__ void __launch_bounds__(PA_THREADS<NWG>, 1)
prefill_attn_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_c, const AttnParams p) {
    constexpr int PA_DQK = CFG::DQK, PA_K_BYTES = CFG::K_BYTES, PA_CST = CFG::CST, PA_OFF_C = CFG::OFF_C, PA_OFF_P = CFG::OFF_P,
                  PA_OFF_BAR = CFG::OFF_BAR, PA_OFF_X = CFG::OFF_X;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t *sm = smem_raw + (base - raw);
    const uint32_t bar0 = base + PA_OFF_BAR;
    auto bar = [&](int i) { return bar0 + 8u * (uint32_t)i; };
    uint32_t *s_tmem = reinterpret_cast<uint32_t *>(sm + PA_OFF_BAR + 8 * PB_COUNT + 8);
    int4 *s_item = reinterpret_cast<int4 *>(sm + PA_OFF_X + 4096);      // ring of 8 items: {number, first tile, end, record}
    // (P stays in shared memory. In the place of the scores it comes from, in tensor memory, the value MMAs are a link of the next
    // scores' chain: 105 -> 117 us for 512 GQA queries after 10488 rows.)
    constexpr int TG = NWG == 4 ? 2 : 1, QK_ISSUERS = NWG == 4 ? 2 : 1;      // groups that share a tile; issuers of the score MMAs
    float *s_m = reinterpret_cast<float *>(sm + PA_OFF_X), *s_l = s_m + 512;              // [4][128] each

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    cwk_pdl_launch();
    cwk_pdl_wait();
    if (NWG == 1 && p.counter[2] == 0) return;                   // the repair pass: the fast form raised no flag
    const int nq = (p.n + PA_QT - 1) / PA_QT;
    const int total = nq * p.nh;
    const int unit = GQA ? (int)blockIdx.x : (int)blockIdx.x >> 1;      // share mode: whose share this block works on (MLA: one half of it)

    if (tid == 0) {
        asm volatile("prefetch.tensormap [%0];" ::"l"(&tm_k) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&tm_c) : "memory");
        for (int i = 0; i < PB_COUNT; i++) {
            // (an arrival per softmax warp; 32 a warp on one barrier are served one after another)
            const bool by_tile = i >= PB_SEMPTY && i < PB_PEMPTY, by_soft = i == PB_QFULL || i == PB_OFREE || i == PB_XM || i == PB_XL;
            mbar_init(bar(i), by_tile ? (uint32_t)(4 * TG) : by_soft ? (uint32_t)(4 * NWG) : i == PB_QEMPTY ? QK_ISSUERS : 1u);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(s_tmem)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *s_tmem;

    // item k of this block, as published by the key producer (w < 0: no more)
    auto read_item = [&](int k, int &w, AttnItem &it) {
        const int4 v = s_item[k & 7];
        w = GQA || v.x < 0 ? v.x : v.x >> 1;
        it = attn_item(max(w, 0), p, nq);
        it.half = GQA ? 0 : v.x & 1;
        it.lo = v.y; it.nt = v.z; it.rec = v.w;
        if (p.shares) it.flag = w + unit;
    };
    auto next_item = [&](int k, int &w, AttnItem &it) -> bool {      // a warp's
        if (!mbar_wait_warp(bar(PB_ITEM + (k & 7)), (uint32_t)((k >> 3) & 1), p.err, 1031)) return false;
        read_item(k, w, it);
        return true;
    };

    if (warp == 0) {
        // ------------------------------------------------------------ item fetcher and TMA producer of the key ring
        if (lane == 0) {
            bool ok = true;
            int kc = 0;                              // key tiles issued so far (ring position and phase run across items)
            const int64_t all = (int64_t)p.head_tiles * p.nh, u0 = p.shares ? share_begin(unit, all, p.shares) : 0,
                          u1 = p.shares ? share_begin(unit + 1, all, p.shares) : 0;
            int sw = 0;                              // share mode: the next item, and where it begins
            int64_t at = 0;
            if (p.shares) {
                sw = (int)u0 / p.head_tiles * nq;
                at = (int)u0 / p.head_tiles * p.head_tiles;
                for (int nt; sw < total && at + (nt = attn_item(sw, p, nq).nt) <= u0; sw++) at += nt;
            }
            for (int k = 0; ok; k++) {
                int w = -1, half = GQA ? 0 : (int)blockIdx.x & 1;
                AttnItem it{};
                if (p.shares) {
                    while (sw < total && at < u1) {
                        it = attn_item(sw, p, nq);
                        const int nt = it.nt;
                        const bool mine = attn_segment(it, sw, unit, at, u0, u1, p);
                        at += nt;
                        sw++;
                        if (mine && (NWG > 1 || p.flags[it.flag] != 0)) { w = sw - 1; break; }      // (the repair pass takes flagged ones only)
                    }
                } else {
                    constexpr int H = GQA ? 1 : 2;    // an item is one of its halves here
                    int hw = atomicAdd(p.counter + (NWG == 1 ? 1 : 0), 1);
                    if (NWG == 1)                     // the repair pass takes flagged items only
                        while (hw < total * H && p.flags[hw / H] == 0) hw = atomicAdd(p.counter + 1, 1);
                    w = hw < total * H ? hw / H : -1;
                    half = hw % H;
                    it = attn_item(max(w, 0), p, nq);
                }
                it.half = half;
                s_item[k & 7] = make_int4(GQA || w < 0 ? w : 2 * w + half, it.lo, it.nt, it.rec);      // the roles of a block stay within a few tiles of each other: 8 slots cannot wrap
                mbar_arrive(bar(PB_ITEM + (k & 7)));
                if (w < 0) break;
                for (int i = it.lo; i < it.nt && ok; i++, kc++) {
                    const int ks = kc % PA_KST, ku = kc / PA_KST;
                    ok = mbar_wait(bar(PB_KEMPTY + ks), (uint32_t)((ku & 1) ^ 1), p.err, 1001);
                    if (!ok) break;
                    const uint32_t full = bar(PB_KFULL + kc % PA_KBAR);
                    mbar_expect_tx(full, PA_K_BYTES);
                    if (GQA) tma_load_3d(base + PA_OFF_K + ks * PA_K_BYTES, &tm_k, 0, i * PA_KT, (it.h / p.group) * (PA_DQK / 64), full);
                    else tma_load_3d(base + PA_OFF_K + ks * PA_K_BYTES, &tm_k, 0, it.h * p.T + i * PA_KT, 0, full);
                }
            }
            if (!ok)        // drain the copies still in flight before leaving
                for (int j = (kc > PA_KST ? kc - PA_KST : 0); j < kc; j++)
                    mbar_wait(bar(PB_KFULL + j % PA_KBAR), (uint32_t)((j / PA_KBAR) & 1), p.err, 1004);
        }
    } else if (warp == 2) {
        // ------------------------------------------------------------ TMA producer of the latent ring (its slots come free much
        // later than the key slots: a thread of its own, so that the keys run ahead)
        if (lane == 0) {
            bool ok = true;
            int cc = 0;
            for (int k = 0; ok; k++) {
                int w;
                AttnItem it;
                ok = mbar_wait(bar(PB_ITEM + (k & 7)), (uint32_t)((k >> 3) & 1), p.err, 1032);
                if (!ok) break;
                read_item(k, w, it);
                if (w < 0) break;
                for (int i = it.lo; i < it.nt && ok; i++, cc++) {
                    const int cs = cc % PA_CST, cu = cc / PA_CST;
                    ok = mbar_wait(bar(PB_CEMPTY + cs), (uint32_t)((cu & 1) ^ 1), p.err, 1002);
                    if (!ok) break;
                    mbar_expect_tx(bar(PB_CFULL + cs), PA_C_BYTES);
                    tma_load_3d(base + PA_OFF_C + cs * PA_C_BYTES, &tm_c, 0, i * PA_KT, (GQA ? it.h / p.group : it.half) * 4, bar(PB_CFULL + cs));
                }
            }
            if (!ok)
                for (int j = (cc > PA_CST ? cc - PA_CST : 0); j < cc; j++)
                    mbar_wait(bar(PB_CFULL + j % PA_CST), (uint32_t)((j / PA_CST) & 1), p.err, 1005);
        }
    } else if (warp == 1 || warp == 4 + 4 * NWG) {
        // ------------------------------------------------------------ MMA issuers of the scores
        // The two products have issuers of their own (this warp and warp 3): a wait on an mbarrier costs a
        // lone thread some 200 cycles even when the phase is long complete, and one thread doing all four
        // waits of a tile in turn was the longest chain of the kernel. So was, after that, the one issuer of the scores: two
        // waits, 12 or 16 MMAs and the commits took it 1650 cycles a tile, of which the tensor pipe works 400 to 500. In the fast
        // form a second one (the last warp) takes every other tile. All lanes run the issuers' loops and one is elected for the
        // MMAs (tc_common.cuh).
        {
            uint32_t patience = WAIT_LIMIT;
            constexpr uint32_t ID_QK = idesc_bf16(128, PA_KT, 0, 0);
            const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
            const uint64_t dK0 = smem_desc(base + PA_OFF_K, 16, 1024);
            const int first = QK_ISSUERS == 2 && warp != 1 ? 1 : 0;
            bool ok = true;
            int kc = 0;                              // score tiles so far
            for (int k = 0; ok; k++) {
                int w;
                AttnItem it;
                ok = next_item(k, w, it);
                if (!ok || w < 0) break;
                const int end = __shfl_sync(0xffffffffu, kc + it.nt - it.lo, 0);
                ok = mbar_wait_warp(bar(PB_QFULL), (uint32_t)(k & 1), p.err, 1011);     // the softmax threads have written the item's query tile into tensor memory
                if (!ok) break;
                tc_fence_after();
                // scores of a tile: S[kc % 2] = Q Kx^T, the 64-wide blocks of the key's dims, four 16-wide steps each
#pragma unroll 1
                for (kc += QK_ISSUERS == 2 ? (kc ^ first) & 1 : 0; kc < end; kc += QK_ISSUERS) {
                    const int ks = kc % PA_KST, sb = kc % PA_SBUF, su = kc / PA_SBUF;
                    mbar_wait_on(bar(PB_KFULL + kc % PA_KBAR), (uint32_t)((kc / PA_KBAR) & 1), p.err, 1012, patience);
                    mbar_wait_on(bar(PB_SEMPTY + sb), (uint32_t)((su & 1) ^ 1), p.err, 1013, patience);
                    tc_fence_after();
                    const uint64_t dK = dK0 + (uint64_t)((ks * PA_K_BYTES) >> 4);
                    if (elect_one()) {
#pragma unroll
                        for (int s = 0; s < PA_DQK / 16; s++)
                            umma_bf16_ts(tm + PA_COL_S + sb * PA_KT, tm + PA_COL_Q + s * 8,       // A: 16 bf16 of every row = 8 TMEM columns per step
                                         dK + (uint64_t)(((s >> 2) * (PA_KT * 128) + (s & 3) * 32) >> 4), ID_QK, s != 0);
                        umma_commit(bar(PB_KEMPTY + ks));
                        umma_commit(bar(PB_SFULL + sb));
                    }
                    __syncwarp();
                }
                kc = end;
                if (elect_one()) umma_commit(bar(PB_QEMPTY));       // the query tile may be replaced once these MMAs are done
                __syncwarp();
            }
            settle(patience != WAIT_LIMIT);
        }
    } else if (warp == 3) {
        // ------------------------------------------------------------ MMA issuer of the values
        {
            uint32_t patience = WAIT_LIMIT;
            constexpr uint32_t ID_PV = idesc_bf16(128, PA_DV, 0, 1);
            const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
            const uint64_t dP0 = smem_desc(base + PA_OFF_P, 16, 1024), dC0 = smem_desc(base + PA_OFF_C, PA_KT * 128, 1024);
            bool ok = true;
            int cc = 0;                              // value tiles issued so far
            for (int k = 0; ok; k++) {
                int w;
                AttnItem it;
                ok = next_item(k, w, it);
                if (!ok || w < 0) break;
                const int tiles = __shfl_sync(0xffffffffu, it.nt - it.lo, 0);
                if (k > 0) {                         // the accumulator of the previous item has been read out
                    ok = mbar_wait_warp(bar(PB_OFREE), (uint32_t)((k - 1) & 1), p.err, 1016);
                    if (!ok) break;
                }
#pragma unroll 1
                for (int i = 0; i < tiles; i++, cc++) {
                    const int cs = cc % PA_CST, cu = cc / PA_CST, pb = cc & 1, pu = cc >> 1;
                    mbar_wait_on(bar(PB_CFULL + cs), (uint32_t)(cu & 1), p.err, 1014, patience);
                    mbar_wait_on(bar(PB_PFULL + pb), (uint32_t)(pu & 1), p.err, 1015, patience);
                    tc_fence_after();
                    // values: O += P lat, P [128 q][64 keys] K-major, lat half [64 keys][256] with the 256 contiguous (MN-major, four 64-wide blocks)
                    const uint64_t dP = dP0 + (uint64_t)((pb * PA_P_BYTES) >> 4), dC = dC0 + (uint64_t)((cs * PA_C_BYTES) >> 4);
                    if (elect_one()) {
#pragma unroll
                        for (int s = 0; s < 4; s++) {
                            const uint32_t acc = s != 0 ? 1u : (uint32_t)(i != 0);
                            umma_bf16(tm + PA_COL_O, dP + (uint64_t)((s * 32) >> 4), dC + (uint64_t)((s * 2048) >> 4), ID_PV, acc);
                        }
                        umma_commit(bar(PB_CEMPTY + cs));
                        umma_commit(bar(PB_PEMPTY + pb));
                    }
                    __syncwarp();
                }
                if (elect_one()) umma_commit(bar(PB_ODONE));
                __syncwarp();
            }
            settle(patience != WAIT_LIMIT);
        }
    } else {
        // ------------------------------------------------------------ softmax, (correction,) epilogue
        // A thread owns query row `row` (= its TMEM lane) and NC of the 64 key columns of its tiles.
        constexpr int NC = PA_KT / TG;
        const int q4 = warp & 3, wg = (warp - 4) >> 2, cg = wg & (TG - 1), odd = wg / TG;      // columns cg * NC .., tiles of parity `odd`
        const int row = q4 * 32 + lane;
        const uint32_t tlane = tmem + ((uint32_t)(q4 * 32) << 16);
        auto arrive = [&](int b) {                   // one for the warp, after every lane's accesses
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(b));
        };
        bool ok = true;
        int tc = 0;                                  // tiles done so far (score buffer, P buffer and their phases run across items)
        for (int k = 0; ok; k++) {
            int w;
            AttnItem it;
            ok = next_item(k, w, it);
            if (!ok || w < 0) break;
            const int q0 = it.q0, h = it.h, half = it.half, nt = it.nt;
            const int64_t tq = p.pos0 + q0 + row;                    // this row's position: keys 0..tq are visible
            auto load_query = [&](int q0_, int h_) { load_query_tile<CFG, NWG, GQA>(p, q0_, h_, row, wg, tlane, [&]() { arrive(PB_QFULL); }); };
            if (k == 0) load_query(q0, h);
            float m = 0.f, l = 0.f;
            // reference exponent of the row: its largest score of the item's first tile, which one pair of groups has. (All arrive:
            // no P is written before the epilogue of the item before has left the P buffers.)
            auto reference = [&]() -> bool {
                arrive(PB_XM);
                if (!mbar_wait_warp(bar(PB_XM), (uint32_t)(k & 1), p.err, 1026)) return false;
                m = fmaxf(s_m[row], s_m[128 + row]);                 // the tile shows every row a key: finite
                return true;
            };
            if (NWG == 4 && (tc & 1) != odd && !reference()) break;
            const int tc0 = tc;
            tc += nt - it.lo;
            for (int d = NWG == 4 ? (tc0 ^ odd) & 1 : 0; d < nt - it.lo; d += NWG == 4 ? 2 : 1) {
                const int i = it.lo + d, sb = (tc0 + d) & 1, su = (tc0 + d) >> 1;      // the tile; its score and P buffers and their use
                ok = mbar_wait_warp(bar(PB_SFULL + sb), (uint32_t)(su & 1), p.err, 1021);   // the TMEM loads below are warp-wide
                if (!ok) break;
                tc_fence_after();
                uint32_t v[NC];
#pragma unroll
                for (int c = 0; c < NC / 16; c++) TMEM_LD16(v, c * 16, tlane + PA_COL_S + sb * PA_KT + cg * NC + c * 16);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                tc_fence_before();
                arrive(PB_SEMPTY + sb);
                const bool whole = (int64_t)i * PA_KT + PA_KT - 1 <= p.pos0 + q0;      // every key of the tile is visible to every row of the item
                const int seen = (int)min(tq - (int64_t)i * PA_KT - cg * NC, (int64_t)PA_KT);      // the thread's keys 0 .. seen are visible
                if (NWG == 4 && i == it.lo) {
                    float mt = -INFINITY;
#pragma unroll
                    for (int j = 0; j < NC; j++) mt = fmaxf(mt, whole || j <= seen ? __uint_as_float(v[j]) * p.scale_log2 : -INFINITY);
                    s_m[cg * 128 + row] = mt;
                    ok = reference();
                    if (!ok) break;
                }
                // exponents relative to the reference: scale, difference and below the sum two at a time
                float s[NC];
                const uint64_t scale2 = pack_f32x2(p.scale_log2, p.scale_log2), minus_m = NWG == 4 ? pack_f32x2(-m, -m) : 0;
#pragma unroll
                for (int j = 0; j < NC; j += 2)
                    unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(v[j]), __uint_as_float(v[j + 1])), scale2, minus_m), s[j], s[j + 1]);
                if (!whole) {
#pragma unroll
                    for (int j = 0; j < NC; j++)
                        if (j > seen) s[j] = -INFINITY;
                }
                float mt = s[0];
#pragma unroll
                for (int j = 1; j + 1 < NC; j += 2) mt = fmaxf(mt, fmaxf(s[j], s[j + 1]));
                mt = fmaxf(mt, s[NC - 1]);
                if (NWG == 4) {
                    if (mt > PA_RANGE) {
                        p.flags[it.flag] = 1;                        // out of the range this form covers: the exact form redoes the item
                        atomicAdd(p.counter + 2, 1);
                    }
                } else {
                    // tcgen05.ld / st are warp-wide instructions: the warp decides together, and a lane that has no
                    // need of it rescales by 1
                    const bool mine = (i != it.lo) && (mt > m + PA_LAZY);
                    if (i == it.lo) m = mt;
                    if (__any_sync(0xffffffffu, mine)) {
                        // some row's scores outran its reference exponent: rescale what it has accumulated. A row is its
                        // thread's TMEM lane; the value MMAs of the previous tile must have finished writing it.
                        ok = mbar_wait_warp(bar(PB_PEMPTY + ((tc0 + d - 1) & 1)), (uint32_t)(((tc0 + d - 1) >> 1) & 1), p.err, 1022);
                        if (!ok) break;
                        tc_fence_after();
                        const float alpha = mine ? exp2f(m - mt) : 1.f;
                        l *= alpha;
                        if (mine) m = mt;
                        for (int c = 0; c < PA_DV / 16; c++) {
                            uint32_t o[16];
                            TMEM_LD16(o, 0, tlane + PA_COL_O + c * 16);
                            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                            for (int j = 0; j < 16; j++) o[j] = __float_as_uint(__uint_as_float(o[j]) * alpha);
                            TMEM_ST16(o, 0, tlane + PA_COL_O + c * 16);
                        }
                        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                    }
                }
                uint32_t pk[NC / 2];
                uint64_t lsum = 0;                                   // two f32 zeros
#pragma unroll
                for (int j = 0; j < NC; j += 2) {
                    const float p0 = exp2f(NWG == 4 ? s[j] : s[j] - m), p1 = exp2f(NWG == 4 ? s[j + 1] : s[j + 1] - m);
                    lsum = add_f32x2(lsum, pack_f32x2(p0, p1));
                    pk[j >> 1] = pack_bf16x2(p0, p1);
                }
                float l0, l1;
                unpack_f32x2(lsum, l0, l1);
                l += l0 + l1;
                // the P buffer of this parity was read by the value MMAs two tiles ago
                ok = mbar_wait_warp(bar(PB_PEMPTY + sb), (uint32_t)((su & 1) ^ 1), p.err, 1023);
                if (!ok) break;
                uint8_t *prow = sm + PA_OFF_P + sb * PA_P_BYTES + row * 128;
#pragma unroll
                for (int c = 0; c < NC / 8; c++)
                    *reinterpret_cast<uint4 *>(prow + (((cg * (NC / 8) + c) ^ (row & 7)) << 4)) = make_uint4(pk[4 * c], pk[4 * c + 1], pk[4 * c + 2], pk[4 * c + 3]);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                tc_fence_before();
                arrive(PB_PFULL + sb);
            }
            if (!ok) break;
            {
                // the next item's query tile: the score MMAs of this item are done with theirs (they precede its last value MMAs)
                int wn;
                AttnItem nx;
                ok = next_item(k + 1, wn, nx);
                if (!ok) break;
                if (wn >= 0) {
                    ok = mbar_wait_warp(bar(PB_QEMPTY), (uint32_t)(k & 1), p.err, 1025);
                    if (!ok) break;
                    tc_fence_after();
                    load_query(nx.q0, nx.h);
                }
            }
            // ---- epilogue of the item: O / l -> bf16 -> out[t][h][half * 256 ..], full lines through a staging tile
            ok = mbar_wait_warp(bar(PB_ODONE), (uint32_t)(k & 1), p.err, 1024);
            if (!ok) break;
            tc_fence_after();
            if (NWG == 4) {                                          // the row's sum is the groups' sums
                s_l[wg * 128 + row] = l;
                arrive(PB_XL);
                ok = mbar_wait_warp(bar(PB_XL), (uint32_t)(k & 1), p.err, 1027);
                if (!ok) break;
                l = (s_l[row] + s_l[128 + row]) + (s_l[256 + row] + s_l[384 + row]);
            }
            if (it.rec >= 0) {                                       // part of an item: its record
                float *rec = p.records + record_of<GQA>(it.rec, half) * PA_RECORD;
                constexpr int CPG = PA_DV / NWG;                     // columns per group
#pragma unroll 1
                for (int c = 0; c < CPG / 16; c++) {
                    const int col = wg * CPG + c * 16;
                    uint32_t o[16];
                    TMEM_LD16(o, 0, tlane + PA_COL_O + col);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int j = 0; j < 4; j++)
                        *reinterpret_cast<uint4 *>(rec + ((int64_t)(col / 4 + j) * PA_QT + row) * 4) = make_uint4(o[4 * j], o[4 * j + 1], o[4 * j + 2], o[4 * j + 3]);
                }
                if (wg == 0) { rec[PA_QT * PA_DV + row] = m; rec[PA_QT * (PA_DV + 1) + row] = l; }
                tc_fence_before();
                arrive(PB_OFREE);
                continue;
            }
            // All groups write out (two of four, 64 columns at a time: 12 k cycles an item with the next query's copy; now 8 k)
            const float inv = l > 0.f ? 1.f / l : 0.f;
            // 2 KB per warp, [32 rows][64 B], in the P buffers: the item's value MMAs are done, and the next item's P is written behind
            // reference(), where all meet. The exact form's warps meet nowhere: each stages in the place of its own rows' P, which
            // no other warp writes.
            uint8_t *stg = sm + PA_OFF_P + (warp - 4) * (NWG == 4 ? 2048 : 32 * 128);
            const int t0w = q0 + q4 * 32;
            constexpr int NCH = PA_DV / 64 / NWG;                     // 64-column chunks per thread
#pragma unroll 1
            for (int c = 0; c < NCH; c++) {
                const int col = (wg * NCH + c) * 64;
                uint32_t o[64];
                TMEM_LD16(o, 0, tlane + PA_COL_O + col);
                TMEM_LD16(o, 16, tlane + PA_COL_O + col + 16);
                TMEM_LD16(o, 32, tlane + PA_COL_O + col + 32);
                TMEM_LD16(o, 48, tlane + PA_COL_O + col + 48);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (c == NCH - 1) {
                    tc_fence_before();
                    arrive(PB_OFREE);                                // the value MMAs of the next item may overwrite the accumulator
                }
#pragma unroll
                for (int u = 0; u < 2; u++) {
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        const uint32_t *x = o + u * 32 + 8 * j;
                        uint4 wv;
                        wv.x = pack_bf16x2(__uint_as_float(x[0]) * inv, __uint_as_float(x[1]) * inv);
                        wv.y = pack_bf16x2(__uint_as_float(x[2]) * inv, __uint_as_float(x[3]) * inv);
                        wv.z = pack_bf16x2(__uint_as_float(x[4]) * inv, __uint_as_float(x[5]) * inv);
                        wv.w = pack_bf16x2(__uint_as_float(x[6]) * inv, __uint_as_float(x[7]) * inv);
                        *reinterpret_cast<uint4 *>(stg + lane * 64 + ((j ^ ((lane >> 1) & 3)) << 4)) = wv;
                    }
                    __syncwarp();
#pragma unroll
                    for (int r = 0; r < 4; r++) {
                        const int rr = r * 8 + (lane >> 2), jj = lane & 3;
                        const uint4 wv = *reinterpret_cast<const uint4 *>(stg + rr * 64 + ((jj ^ ((rr >> 1) & 3)) << 4));
                        if (t0w + rr < p.n)
                            *reinterpret_cast<uint4 *>(p.out + ((int64_t)(t0w + rr) * p.nh + h) * (GQA ? PA_DV : PA_L) + half * PA_DV + col + u * 32 + jj * 8) = wv;
                    }
                    __syncwarp();
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

// ---- the fast form of the MLA prompt: a pair of CTAs shares its scores ---------------------------------------------------
// Both halves of the value columns want the same scores, 192 wide, and their exponentials: done by each half for itself they are
// 384 of 896 multiply-adds per (query, key, head), and a whole prompt is at the power cap. Here the halves are the two CTAs of a
// cluster. The tiles of all items have running numbers T; the CTA with rank T & 1 forms tile T's scores and P, and P goes to the other by a bulk copy
// between their shared memories, so that each does half the scores and all of its values. (The first tile of an item gives the
// rows' reference exponents: both form its scores, one uses them. The row sums are exchanged at the item's end.)
//
// 4096 tokens (whole prompt) 1555 -> 1471 us, 509 after 3001 349 -> 330. With the copies issued by the values' issuer, in the order of
// the tiles, each waited for the peer's copy of the tile before: 2.7 k cycles a tile, 1792 us.
//
// P lies in four buffers, tile T in buffer T % 4 of both CTAs: those of its own tiles a CTA's softmax writes, the others the
// peer fills (an even number: a role that looks at own tiles only sees every phase of their barriers; six of them beside two latent
// stages instead of three: 1490 and 338 us). A buffer is free for tile T + 4 when the value MMAs of tile T are done in BOTH CTAs, and
// both tell the CTA whose tile it is, which alone writes tile T + 4, and it alone: every arrival from the other CTA is then one that
// somebody waits for, the last two tiles' before the epilogue, and none is under way when a CTA leaves. There are eight of these
// barriers, T % 8: the two softmax sets of a CTA may be
// an own tile apart, and with four a set could wait for a phase whose predecessor is still open, which a parity wait cannot tell
// from the one after. tests/test_prefill_pair_protocol.py walks the protocol.
template <class CFG>
struct PrCfg {
    static constexpr int KST = 2, CST = 3;
    static constexpr int OFF_C = KST * CFG::K_BYTES, OFF_P = OFF_C + CST * PA_C_BYTES, OFF_BAR = OFF_P + 4 * PA_P_BYTES, OFF_X = OFF_BAR + 512;
    static constexpr int SMEM = OFF_X + 2 * 2048 + 4 * 512 + 128 + 1024;      // maxima [4][128], sums [4][128], row sums here and there [2][128] each, 8 items
    static_assert(SMEM <= 232448, "shared-memory budget");
};
constexpr int PR_THREADS = 672;      // keys, scores, latents, values | 16 softmax warps | sender of P
enum { PR_QFULL = 0, PR_KFULL, PR_KEMPTY = PR_KFULL + 2, PR_CFULL = PR_KEMPTY + 2, PR_CEMPTY = PR_CFULL + 3, PR_SFULL = PR_CEMPTY + 3, PR_SEMPTY = PR_SFULL + 2,
       PR_PFULL = PR_SEMPTY + 2, PR_PEMPTY = PR_PFULL + 4, PR_ODONE = PR_PEMPTY + 8, PR_QEMPTY, PR_OFREE, PR_XM, PR_XL, PR_PEER, PR_ITEM = PR_PEER + 2,
       PR_COUNT = PR_ITEM + 8 };
static_assert(8 * PR_COUNT + 16 <= 512, "barriers");

// shared memory of this CTA to the same offset in CTA `peer` of the cluster, its bytes counted at that CTA's barrier (multiples of 16 bytes)
__device__ __forceinline__ void copy_to_peer(uint32_t addr, uint32_t bytes, uint32_t peer_addr, uint32_t peer_bar) {
    asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(peer_addr), "r"(addr), "r"(bytes), "r"(peer_bar)
                 : "memory");
}
// completion of this CTA's MMAs so far, at the same barrier in the CTAs of the cluster that `ctas` has bits for
__device__ __forceinline__ void umma_commit_to(uint32_t bar, int ctas) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((uint16_t)ctas) : "memory");
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PR_THREADS, 1)
prefill_pair_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_c, const AttnParams p) {
    using CFG = PaMla;
    using L = PrCfg<CFG>;
    constexpr int NC = PA_KT / 2;                            // key columns per softmax thread
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t *sm = smem_raw + (base - raw);
    const uint32_t bar0 = base + L::OFF_BAR;
    auto bar = [&](int i) { return bar0 + 8u * (uint32_t)i; };
    uint32_t *s_tmem = reinterpret_cast<uint32_t *>(sm + L::OFF_BAR + 8 * PR_COUNT + 8);
    float *s_m = reinterpret_cast<float *>(sm + L::OFF_X), *s_l = s_m + 512, *s_sum = s_l + 512, *s_peer = s_sum + 256;
    int4 *s_item = reinterpret_cast<int4 *>(s_peer + 256);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rank = (int)cluster_rank(), unit = (int)blockIdx.x >> 1, units = (int)gridDim.x >> 1;
    cwk_pdl_launch();
    cwk_pdl_wait();
    const int nq = (p.n + PA_QT - 1) / PA_QT, total = nq * p.nh;

    if (tid == 0) {
        asm volatile("prefetch.tensormap [%0];" ::"l"(&tm_k) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&tm_c) : "memory");
        for (int i = 0; i < PR_COUNT; i++) {
            uint32_t count = 1;
            if (i == PR_QFULL || i == PR_OFREE || i == PR_XM || i == PR_XL) count = 16;                  // every softmax warp
            if (i == PR_SEMPTY || i == PR_SEMPTY + 1) count = 8;                                         // the warps of a set
            if (i >= PR_PFULL && i < PR_PEMPTY) count = ((i - PR_PFULL) & 1) == rank ? 8 : 1;            // ... or the announcement of the peer's copy
            if (i == PR_PEER || i == PR_PEER + 1) count = 4;                                             // the announcements of the warps that exchange row sums
            if (i >= PR_PEMPTY && i < PR_ODONE) count = 2;                                               // the value MMAs of both CTAs (own tiles' barriers)
            mbar_init(bar(i), count);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(s_tmem)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();                                          // the peer's barriers are there
    tc_fence_after();
    const uint32_t tmem = *s_tmem;

    // item k of this pair, as published by the key producer (w < 0: no more); both CTAs come to the same items by themselves
    auto read_item = [&](int k, int &w, AttnItem &it) {
        const int4 v = s_item[k & 7];
        w = v.x;
        it = attn_item(max(w, 0), p, nq);
        it.half = rank;
        it.lo = v.y; it.nt = v.z; it.rec = v.w;
        if (p.shares) it.flag = w + unit;
    };
    auto next_item = [&](int k, int &w, AttnItem &it) -> bool {      // a warp's
        if (!mbar_wait_warp(bar(PR_ITEM + (k & 7)), (uint32_t)((k >> 3) & 1), p.err, 1431)) return false;
        read_item(k, w, it);
        return true;
    };
    // the tiles of an item whose first has number T: how many this CTA forms the scores of (the first, and its own), and the i-th of them
    auto scored = [&](int T, int tiles) { const int f = ((T + 1) & 1) == rank ? 1 : 2; return tiles > f ? 1 + (tiles - f + 1) / 2 : 1; };
    auto nth = [&](int T, int e) { return e == 0 ? 0 : (((T + 1) & 1) == rank ? 1 : 2) + 2 * (e - 1); };

    if (warp == 0) {
        // ------------------------------------------------------------ item fetcher and TMA producer of the key ring
        if (lane == 0) {
            bool ok = true;
            int kc = 0, T = 0;                       // key tiles issued so far; number of the item's first tile
            const int64_t all = (int64_t)p.head_tiles * p.nh, u0 = p.shares ? share_begin(unit, all, p.shares) : 0, u1 = p.shares ? share_begin(unit + 1, all, p.shares) : 0;
            int sw = 0;                              // share mode: the next item, and where it begins
            int64_t at = 0;
            if (p.shares) {
                sw = (int)u0 / p.head_tiles * nq;
                at = (int)u0 / p.head_tiles * p.head_tiles;
                for (int nt; sw < total && at + (nt = attn_item(sw, p, nq).nt) <= u0; sw++) at += nt;
            }
            for (int k = 0; ok; k++) {
                int w = -1;
                AttnItem it{};
                if (p.shares) {
                    while (sw < total && at < u1) {
                        it = attn_item(sw, p, nq);
                        const int nt = it.nt;
                        const bool mine = attn_segment(it, sw, unit, at, u0, u1, p);
                        at += nt;
                        sw++;
                        if (mine) { w = sw - 1; break; }
                    }
                } else {
                    // in rounds, there and back: a pair that had the longer items of one round has the shorter ones of the next
                    w = k * units + ((k & 1) ? units - 1 - unit : unit);
                    if (w >= total) w = -1;
                    it = attn_item(max(w, 0), p, nq);
                }
                s_item[k & 7] = make_int4(w, it.lo, it.nt, it.rec);      // the roles of a block stay within a few tiles of each other: 8 slots cannot wrap
                mbar_arrive(bar(PR_ITEM + (k & 7)));
                if (w < 0) break;
                const int tiles = it.nt - it.lo, mine = scored(T, tiles);
                for (int e = 0; e < mine && ok; e++, kc++) {
                    const int ks = kc % L::KST;
                    ok = mbar_wait(bar(PR_KEMPTY + ks), (uint32_t)(((kc / L::KST) & 1) ^ 1), p.err, 1401);
                    if (!ok) break;
                    mbar_expect_tx(bar(PR_KFULL + ks), CFG::K_BYTES);
                    tma_load_3d(base + ks * CFG::K_BYTES, &tm_k, 0, it.h * p.T + (it.lo + nth(T, e)) * PA_KT, 0, bar(PR_KFULL + ks));
                }
                T += tiles;
            }
            if (!ok)        // drain the copies still in flight before leaving
                for (int j = max(0, kc - L::KST); j < kc; j++) mbar_wait(bar(PR_KFULL + j % L::KST), (uint32_t)((j / L::KST) & 1), p.err, 1404);
        }
    } else if (warp == 2) {
        // ------------------------------------------------------------ TMA producer of the latent ring: every tile, this CTA's half; announces the peer's P
        if (lane == 0) {
            bool ok = true;
            int cc = 0;
            for (int k = 0; ok; k++) {
                int w;
                AttnItem it;
                ok = mbar_wait(bar(PR_ITEM + (k & 7)), (uint32_t)((k >> 3) & 1), p.err, 1432);
                if (!ok) break;
                read_item(k, w, it);
                if (w < 0) break;
                for (int i = it.lo; i < it.nt && ok; i++, cc++) {
                    const int cs = cc % L::CST;
                    ok = mbar_wait(bar(PR_CEMPTY + cs), (uint32_t)(((cc / L::CST) & 1) ^ 1), p.err, 1402);
                    if (!ok) break;
                    // the P of the peer's tiles (whose copy may be here before it is announced): what was in its buffer before has been
                    // multiplied, since the values of tile cc - CST have been
                    if ((cc & 1) != rank) mbar_expect_tx(bar(PR_PFULL + (cc & 3)), PA_P_BYTES);
                    mbar_expect_tx(bar(PR_CFULL + cs), PA_C_BYTES);
                    tma_load_3d(base + L::OFF_C + cs * PA_C_BYTES, &tm_c, 0, i * PA_KT, rank * 4, bar(PR_CFULL + cs));
                }
            }
            if (!ok)
                for (int j = max(0, cc - L::CST); j < cc; j++) mbar_wait(bar(PR_CFULL + j % L::CST), (uint32_t)((j / L::CST) & 1), p.err, 1405);
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer of the scores
        uint32_t patience = WAIT_LIMIT;
        constexpr uint32_t ID_QK = idesc_bf16(128, PA_KT, 0, 0);
        const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
        const uint64_t dK0 = smem_desc(base, 16, 1024);
        bool ok = true;
        int kc = 0, T = 0;
        for (int k = 0; ok; k++) {
            int w;
            AttnItem it;
            ok = next_item(k, w, it);
            if (!ok || w < 0) break;
            const int tiles = __shfl_sync(0xffffffffu, it.nt - it.lo, 0), mine = scored(T, tiles);
            ok = mbar_wait_warp(bar(PR_QFULL), (uint32_t)(k & 1), p.err, 1411);     // the softmax threads have written the item's query tile into tensor memory
            if (!ok) break;
            tc_fence_after();
#pragma unroll 1
            for (int e = 0; e < mine; e++, kc++) {
                const int ks = kc % L::KST, sb = kc & 1;
                mbar_wait_on(bar(PR_KFULL + ks), (uint32_t)((kc / L::KST) & 1), p.err, 1412, patience);
                mbar_wait_on(bar(PR_SEMPTY + sb), (uint32_t)(((kc >> 1) & 1) ^ 1), p.err, 1413, patience);
                tc_fence_after();
                const uint64_t dK = dK0 + (uint64_t)((ks * CFG::K_BYTES) >> 4);
                if (elect_one()) {
#pragma unroll
                    for (int s = 0; s < CFG::DQK / 16; s++)
                        umma_bf16_ts(tm + PA_COL_S + sb * PA_KT, tm + PA_COL_Q + s * 8,       // A: 16 bf16 of every row = 8 TMEM columns per step
                                     dK + (uint64_t)(((s >> 2) * (PA_KT * 128) + (s & 3) * 32) >> 4), ID_QK, s != 0);
                    umma_commit(bar(PR_KEMPTY + ks));
                    umma_commit(bar(PR_SFULL + sb));
                }
                __syncwarp();
            }
            if (elect_one()) umma_commit(bar(PR_QEMPTY));       // the query tile may be replaced once these MMAs are done
            __syncwarp();
            T += tiles;
        }
        settle(patience != WAIT_LIMIT);
    } else if (warp == 3) {
        // ------------------------------------------------------------ MMA issuer of the values
        uint32_t patience = WAIT_LIMIT;
        constexpr uint32_t ID_PV = idesc_bf16(128, PA_DV, 0, 1);
        const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
        const uint64_t dP0 = smem_desc(base + L::OFF_P, 16, 1024), dC0 = smem_desc(base + L::OFF_C, PA_KT * 128, 1024);
        bool ok = true;
        int T = 0, cs = 0, cu = 0;                   // tile, value stage and its use
        for (int k = 0; ok; k++) {
            int w;
            AttnItem it;
            ok = next_item(k, w, it);
            if (!ok || w < 0) break;
            const int tiles = __shfl_sync(0xffffffffu, it.nt - it.lo, 0);
            if (k > 0) {                         // the accumulator of the previous item has been read out
                ok = mbar_wait_warp(bar(PR_OFREE), (uint32_t)((k - 1) & 1), p.err, 1416);
                if (!ok) break;
            }
#pragma unroll 1
            for (int i = 0; i < tiles; i++, T++) {
                const int pb = T & 3;
                mbar_wait_on(bar(PR_CFULL + cs), (uint32_t)(cu & 1), p.err, 1414, patience);
                mbar_wait_on(bar(PR_PFULL + pb), (uint32_t)((T >> 2) & 1), p.err, 1415, patience);
                tc_fence_after();
                const uint64_t dP = dP0 + (uint64_t)((pb * PA_P_BYTES) >> 4), dC = dC0 + (uint64_t)((cs * PA_C_BYTES) >> 4);
                if (elect_one()) {
                    // O += P lat, P [128 q][64 keys] K-major, lat half [64 keys][256] with the 256 contiguous (MN-major, four 64-wide blocks)
#pragma unroll
                    for (int s = 0; s < 4; s++)
                        umma_bf16(tm + PA_COL_O, dP + (uint64_t)((s * 32) >> 4), dC + (uint64_t)((s * 2048) >> 4), ID_PV, s != 0 ? 1u : (uint32_t)(i != 0));
                    umma_commit(bar(PR_CEMPTY + cs));
                    umma_commit_to(bar(PR_PEMPTY + (T & 7)), 1 << (T & 1));
                }
                __syncwarp();
                if (++cs == L::CST) { cs = 0; cu++; }
            }
            if (elect_one()) umma_commit(bar(PR_ODONE));
            __syncwarp();
        }
        settle(patience != WAIT_LIMIT);
    } else if (warp == 20) {
        // ------------------------------------------------------------ sender of this CTA's P: as soon as it is there, whatever the values
        // wait for (in the values' issuer a tile's copy waited for the peer's copy of the tile before: 2.7 k cycles a tile)
        const uint32_t peer_p = cluster_addr(base + L::OFF_P, (uint32_t)(rank ^ 1)), peer_bar0 = cluster_addr(bar(PR_PFULL), (uint32_t)(rank ^ 1));
        if (lane == 0) {
            bool ok = true;
            int T = 0;
            for (int k = 0; ok; k++) {
                int w;
                AttnItem it;
                ok = mbar_wait(bar(PR_ITEM + (k & 7)), (uint32_t)((k >> 3) & 1), p.err, 1433);
                if (!ok) break;
                read_item(k, w, it);
                if (w < 0) break;
                const int end = T + it.nt - it.lo;
                for (T += (T ^ rank) & 1; T < end && ok; T += 2) {
                    const int pb = T & 3;
                    ok = mbar_wait(bar(PR_PFULL + pb), (uint32_t)((T >> 2) & 1), p.err, 1417);
                    if (ok) copy_to_peer(base + L::OFF_P + pb * PA_P_BYTES, PA_P_BYTES, peer_p + pb * PA_P_BYTES, peer_bar0 + 8u * (uint32_t)pb);
                }
                T = end;
            }
            settle(!ok);
        }
    } else {
        // ------------------------------------------------------------ softmax, epilogue
        // A thread owns query row `row` (= its TMEM lane) and NC of the 64 key columns of its tiles; two groups have a tile between
        // them, two sets of groups the scored tiles in turn.
        const int q4 = warp & 3, wg = (warp - 4) >> 2, cg = wg & 1, set = wg >> 1;
        const int row = q4 * 32 + lane;
        const uint32_t tlane = tmem + ((uint32_t)(q4 * 32) << 16);
        const uint32_t peer_sum = cluster_addr(smem_u32(s_peer), (uint32_t)(rank ^ 1)), peer_bar0 = cluster_addr(bar(PR_PEER), (uint32_t)(rank ^ 1));
        auto arrive = [&](int b) {                   // one for the warp, after every lane's accesses
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(b));
        };
        auto buffer_free = [&](int T) {              // P buffer T % 4 is free for tile T: both CTAs are done with tile T - 4
            return T < 4 || mbar_wait_warp(bar(PR_PEMPTY + ((T - 4) & 7)), (uint32_t)(((T - 4) >> 3) & 1), p.err, 1423);
        };
        bool ok = true;
        int kc = 0, T = 0;                           // scored tiles so far (score buffer and its phase); number of the item's first tile
        for (int k = 0; ok; k++) {
            int w;
            AttnItem it;
            ok = next_item(k, w, it);
            if (!ok || w < 0) break;
            const int q0 = it.q0, h = it.h, tiles = it.nt - it.lo, mine = scored(T, tiles);
            const int64_t tq = p.pos0 + q0 + row;                    // this row's position: keys 0..tq are visible
            if (k == 0) load_query_tile<CFG, 4, false>(p, q0, h, row, wg, tlane, [&]() { arrive(PR_QFULL); });
            float m = 0.f, l = 0.f;
            // reference exponent of the row: its largest score of the item's first tile, which one set has. (All arrive: no P is written
            // before the epilogue of the item before has left the P buffers.)
            auto reference = [&]() -> bool {
                arrive(PR_XM);
                if (!mbar_wait_warp(bar(PR_XM), (uint32_t)(k & 1), p.err, 1426)) return false;
                m = fmaxf(s_m[row], s_m[128 + row]);                 // the tile shows every row a key: finite
                return true;
            };
            if ((kc & 1) != set && !reference()) break;
            for (int e = (kc ^ set) & 1; e < mine; e += 2) {
                const int d = nth(T, e), i = it.lo + d, sb = (kc + e) & 1, su = (kc + e) >> 1;
                ok = mbar_wait_warp(bar(PR_SFULL + sb), (uint32_t)(su & 1), p.err, 1421);   // the TMEM loads below are warp-wide
                if (!ok) break;
                tc_fence_after();
                uint32_t v[NC];
                TMEM_LD16(v, 0, tlane + PA_COL_S + sb * PA_KT + cg * NC);
                TMEM_LD16(v, 16, tlane + PA_COL_S + sb * PA_KT + cg * NC + 16);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                tc_fence_before();
                arrive(PR_SEMPTY + sb);
                const bool whole = (int64_t)i * PA_KT + PA_KT - 1 <= p.pos0 + q0;      // every key of the tile is visible to every row of the item
                const int seen = (int)min(tq - (int64_t)i * PA_KT - cg * NC, (int64_t)PA_KT);      // the thread's keys 0 .. seen are visible
                if (e == 0) {
                    float mt = -INFINITY;
#pragma unroll
                    for (int j = 0; j < NC; j++) mt = fmaxf(mt, whole || j <= seen ? __uint_as_float(v[j]) * p.scale_log2 : -INFINITY);
                    s_m[cg * 128 + row] = mt;
                    ok = reference();
                    if (!ok) break;
                    if ((T & 1) != rank) continue;                   // the peer's tile
                }
                // exponents relative to the reference: scale, difference and below the sum two at a time
                float s[NC];
                const uint64_t scale2 = pack_f32x2(p.scale_log2, p.scale_log2), minus_m = pack_f32x2(-m, -m);
#pragma unroll
                for (int j = 0; j < NC; j += 2)
                    unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(v[j]), __uint_as_float(v[j + 1])), scale2, minus_m), s[j], s[j + 1]);
                if (!whole) {
#pragma unroll
                    for (int j = 0; j < NC; j++)
                        if (j > seen) s[j] = -INFINITY;
                }
                float mt = s[0];
#pragma unroll
                for (int j = 1; j + 1 < NC; j += 2) mt = fmaxf(mt, fmaxf(s[j], s[j + 1]));
                mt = fmaxf(mt, s[NC - 1]);
                if (mt > PA_RANGE) {
                    p.flags[it.flag] = 1;                            // out of the range this form covers: the exact form redoes the item
                    atomicAdd(p.counter + 2, 1);
                }
                uint32_t pk[NC / 2];
                uint64_t lsum = 0;                                   // two f32 zeros
#pragma unroll
                for (int j = 0; j < NC; j += 2) {
                    const float p0 = exp2f(s[j]), p1 = exp2f(s[j + 1]);
                    lsum = add_f32x2(lsum, pack_f32x2(p0, p1));
                    pk[j >> 1] = pack_bf16x2(p0, p1);
                }
                float l0, l1;
                unpack_f32x2(lsum, l0, l1);
                l += l0 + l1;
                ok = buffer_free(T + d);
                if (!ok) break;
                uint8_t *prow = sm + L::OFF_P + ((T + d) & 3) * PA_P_BYTES + row * 128;
#pragma unroll
                for (int c = 0; c < NC / 8; c++)
                    *reinterpret_cast<uint4 *>(prow + (((cg * (NC / 8) + c) ^ (row & 7)) << 4)) = make_uint4(pk[4 * c], pk[4 * c + 1], pk[4 * c + 2], pk[4 * c + 3]);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                arrive(PR_PFULL + ((T + d) & 3));
            }
            if (!ok) break;
            kc += mine;
            T += tiles;
            {
                // the next item's query tile: the score MMAs of this item are done with theirs (they precede its last value MMAs)
                int wn;
                AttnItem nx;
                ok = next_item(k + 1, wn, nx);
                if (!ok) break;
                if (wn >= 0) {
                    ok = mbar_wait_warp(bar(PR_QEMPTY), (uint32_t)(k & 1), p.err, 1425);
                    if (!ok) break;
                    tc_fence_after();
                    load_query_tile<CFG, 4, false>(p, nx.q0, nx.h, row, wg, tlane, [&]() { arrive(PR_QFULL); });
                }
            }
            // ---- the row's sum: this CTA's four groups', then the peer's
            s_l[wg * 128 + row] = l;
            arrive(PR_XL);
            ok = mbar_wait_warp(bar(PR_XL), (uint32_t)(k & 1), p.err, 1427);
            if (!ok) break;
            if (wg == 0) {
                // (each warp its own rows': a barrier of the four would be waited for without limit where one of them has given up)
                s_sum[(k & 1) * 128 + row] = (s_l[row] + s_l[128 + row]) + (s_l[256 + row] + s_l[384 + row]);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) {
                    mbar_expect_tx(bar(PR_PEER + (k & 1)), 128);
                    copy_to_peer(smem_u32(s_sum + (k & 1) * 128 + row), 128, peer_sum + (k & 1) * 512 + row * 4, peer_bar0 + 8u * (uint32_t)(k & 1));
                }
            }
            l = (s_l[row] + s_l[128 + row]) + (s_l[256 + row] + s_l[384 + row]);
            // ---- epilogue of the item: O / l -> bf16 -> out[t][h][rank * 256 ..], through staging tiles in the buffers of this CTA's
            // own P (the peer may be filling the others): free when both CTAs are done with the last two own tiles
            ok = mbar_wait_warp(bar(PR_PEER + (k & 1)), (uint32_t)((k >> 1) & 1), p.err, 1428);
            if (ok) ok = mbar_wait_warp(bar(PR_ODONE), (uint32_t)(k & 1), p.err, 1424);
            const int next_own = T + ((T & 1) == rank ? 0 : 1);      // the own tile after this item, and the one behind it: in these buffers
            if (ok) ok = buffer_free(next_own);
            if (ok) ok = buffer_free(next_own + 2);
            if (!ok) break;
            tc_fence_after();
            l += s_peer[(k & 1) * 128 + row];
            constexpr int CPG = PA_DV / 4;                           // columns per group
            uint32_t o[CPG];
            TMEM_LD16(o, 0, tlane + PA_COL_O + wg * CPG);
            TMEM_LD16(o, 16, tlane + PA_COL_O + wg * CPG + 16);
            TMEM_LD16(o, 32, tlane + PA_COL_O + wg * CPG + 32);
            TMEM_LD16(o, 48, tlane + PA_COL_O + wg * CPG + 48);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            tc_fence_before();
            arrive(PR_OFREE);                                        // the value MMAs of the next item may overwrite the accumulator
            if (it.rec >= 0) {                                       // part of an item: its record
                float *rec = p.records + record_of<false>(it.rec, rank) * PA_RECORD;
#pragma unroll
                for (int j = 0; j < CPG / 4; j++)
                    *reinterpret_cast<uint4 *>(rec + ((int64_t)(wg * (CPG / 4) + j) * PA_QT + row) * 4) = make_uint4(o[4 * j], o[4 * j + 1], o[4 * j + 2], o[4 * j + 3]);
                if (wg == 0) { rec[PA_QT * PA_DV + row] = m; rec[PA_QT * (PA_DV + 1) + row] = l; }
                continue;
            }
            const float inv = l > 0.f ? 1.f / l : 0.f;
            uint8_t *stg = sm + L::OFF_P + ((warp - 4) < 8 ? rank : rank + 2) * PA_P_BYTES + ((warp - 4) & 7) * 2048;      // 2 KB per warp: [32 rows][64 B]
            const int t0w = q0 + q4 * 32;
#pragma unroll
            for (int u = 0; u < 2; u++) {
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const uint32_t *x = o + u * 32 + 8 * j;
                    uint4 wv;
                    wv.x = pack_bf16x2(__uint_as_float(x[0]) * inv, __uint_as_float(x[1]) * inv);
                    wv.y = pack_bf16x2(__uint_as_float(x[2]) * inv, __uint_as_float(x[3]) * inv);
                    wv.z = pack_bf16x2(__uint_as_float(x[4]) * inv, __uint_as_float(x[5]) * inv);
                    wv.w = pack_bf16x2(__uint_as_float(x[6]) * inv, __uint_as_float(x[7]) * inv);
                    *reinterpret_cast<uint4 *>(stg + lane * 64 + ((j ^ ((lane >> 1) & 3)) << 4)) = wv;
                }
                __syncwarp();
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    const int rr = r * 8 + (lane >> 2), jj = lane & 3;
                    const uint4 wv = *reinterpret_cast<const uint4 *>(stg + rr * 64 + ((jj ^ ((rr >> 1) & 3)) << 4));
                    if (t0w + rr < p.n)
                        *reinterpret_cast<uint4 *>(p.out + ((int64_t)(t0w + rr) * p.nh + h) * PA_L + rank * PA_DV + wg * CPG + u * 32 + jj * 8) = wv;
                }
                __syncwarp();
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();                                          // a CTA's copies and commits to the other have arrived: each was waited for there
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

// Share mode: joins the records of an item that more than one share has a part of. Grid (shares, PA_DV / 32, halves), a row per thread:
// the blocks of share g do the item that its end is the first to cut, if there is one (a grid over all items, most of
// which are whole, took 20 us for 512 of them). 32 columns a thread and 32-bit arithmetic on the shares: 64 items of 512 GQA
// queries after 10488 rows, 39 MB of records, 12.8 -> 8.9 us (sixteen columns and 64-bit divisions before; asking for the next
// segment's columns before the addition of this one's: 10.4, in registers that blocks then lack).
constexpr int PA_MC = 32;                                            // columns per thread
template <bool GQA>
__global__ void __launch_bounds__(128) attn_merge_kernel(const AttnParams p) {
    cwk_pdl_launch();
    const int nq = (p.n + PA_QT - 1) / PA_QT, row = threadIdx.x, c0 = (int)blockIdx.y * PA_MC, half = blockIdx.z;
    const int all = p.head_tiles * p.nh;
    int g = blockIdx.x;
    const int u0 = (int)share_begin(g, all, p.shares), u1 = (int)share_begin(g + 1, all, p.shares);
    int w = u1 / p.head_tiles * nq;                                  // the item with tile u1
    int at = u1 / p.head_tiles * p.head_tiles;
    AttnItem it = attn_item(w, p, nq);
    while (u1 < all && at + it.nt <= u1) {
        at += it.nt;
        it = attn_item(++w, p, nq);
    }
    const bool mine = u1 < all && u1 > at && attn_cut(u1 - at, it, p) > 0 && !(u0 > at && attn_cut(u0 - at, it, p) > 0);
    const int g1 = (int)(((int64_t)(at + it.nt) * p.shares - 1) / all);      // the block that has the item's last tile
    cwk_pdl_wait();                                                  // (in every block: the kernel after this one relies on it)
    if (!mine) return;
    float4 v[PA_MC / 4];
    float ms = 0.f, ls = 0.f;
    // the next segment from block g on
    auto fetch = [&]() {
        for (; g <= g1; g++) {
            AttnItem seg = it;
            if (!attn_segment(seg, w, g, at, share_begin(g, all, p.shares), share_begin(g + 1, all, p.shares), p)) continue;
            const float *rec = p.records + record_of<GQA>(seg.rec, half) * PA_RECORD;
#pragma unroll
            for (int j = 0; j < PA_MC / 4; j++) v[j] = *reinterpret_cast<const float4 *>(rec + ((int64_t)(c0 / 4 + j) * PA_QT + row) * 4);
            ms = rec[PA_QT * PA_DV + row];
            ls = rec[PA_QT * (PA_DV + 1) + row];
            g++;
            return true;
        }
        return false;
    };
    float m = -INFINITY, l = 0.f, o[PA_MC] = {};
    for (bool more = fetch(); more;) {
        const float mn = fmaxf(m, ms), a = exp2f(m - mn), b = exp2f(ms - mn);      // (ms is finite; the first time a is 0)
        m = mn;
        l = l * a + ls * b;
#pragma unroll
        for (int j = 0; j < PA_MC / 4; j++) {
            o[4 * j] = o[4 * j] * a + v[j].x * b; o[4 * j + 1] = o[4 * j + 1] * a + v[j].y * b;
            o[4 * j + 2] = o[4 * j + 2] * a + v[j].z * b; o[4 * j + 3] = o[4 * j + 3] * a + v[j].w * b;
        }
        more = fetch();
    }
    if (it.q0 + row >= p.n) return;
    const float inv = l > 0.f ? 1.f / l : 0.f;
    uint32_t r[PA_MC / 2];
#pragma unroll
    for (int j = 0; j < PA_MC / 2; j++) r[j] = pack_bf16x2(o[2 * j] * inv, o[2 * j + 1] * inv);
    uint4 *dst = reinterpret_cast<uint4 *>(p.out + ((int64_t)(it.q0 + row) * p.nh + it.h) * (GQA ? PA_DV : PA_L) + half * PA_DV + c0);
#pragma unroll
    for (int j = 0; j < PA_MC / 8; j++) dst[j] = make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
}

// The attention grid of both shapes: the fast form, the repair pass, and in share mode the merge. Shares where the longest block (or
// pair) of item-by-item dealing would have more than PA_MERGE_TILES key tiles above an equal share: what the records, their merge and
// its launch cost. GQA, dealt and shared, us, keys and values from memory (16 query heads, 4 KV heads of 256):
//   512 queries after 1500 (19 tiles above the share) 39.5 / 45.5, after 2500 (28) 51.4 / 51.4, after 4000 (41) 68 / 60
//   128 queries after 1500 (23) 37.0 / 41.3, after 2000 (30) 42.6 / 41.5, after 4000 (57) 66 / 45
//   700 queries after 3000 (23) 57.1 / 62.9, after 4000 (28) 68.7 / 70.1, after 6000 (39) 91 / 86
// MLA: more, and a quarter of the share at least: dealt out item by item, the query tiles of a head run at the same time and read its
// keys from memory once, in shares one after the other. Up to the attention, dealt and shared (tiles above the share, of the share):
//   64 heads: 200 queries after 6000 (26 of 164) 258 / 272, 256 after 14000 (60 of 384) 482 / 496, 300 after 20000 (127 of 815) 841 / 867
//   48 heads: 128 after 3000 (17 of 32) 131 / 138, 128 after 8000 (45 of 82) 228 / 221, 256 after 8000 (90 of 166) 303 / 280
//   32 heads: 128 after 3000 (28 of 21) 112 / 115, 128 after 8000 (72 of 55) 184 / 162;  16: 128 after 3000 (38 of 11) 97 / 99, 256 after 8000 (73 of 56) 156 / 137
constexpr int PA_MERGE_TILES = 28, PR_MERGE_TILES = 40;
template <class CFG, bool GQA>
int attn_launch(cwk_ctx *ctx, AttnParams ap, const CUtensorMap &tm_k, const CUtensorMap &tm_c, int exact_only) {
    static bool attr_set[16] = {false};
    if (!attr_set[ctx->device & 15]) {
        CWK_CUDA(ctx, cudaFuncSetAttribute(prefill_attn_kernel<1, CFG, GQA>, cudaFuncAttributeMaxDynamicSharedMemorySize, CFG::SMEM));
        if constexpr (GQA) CWK_CUDA(ctx, cudaFuncSetAttribute(prefill_attn_kernel<4, CFG, GQA>, cudaFuncAttributeMaxDynamicSharedMemorySize, CFG::SMEM));
        else CWK_CUDA(ctx, cudaFuncSetAttribute(prefill_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, PrCfg<CFG>::SMEM));
        attr_set[ctx->device & 15] = true;
    }
    constexpr int H = GQA ? 1 : 2;                                   // blocks that work on an item together
    const int nq = (ap.n + PA_QT - 1) / PA_QT, total = nq * ap.nh, G = ctx->sm_count / H;
    auto tiles = [&](int qtile) { return (ap.pos0 + std::min((int64_t)(qtile + 1) * PA_QT, (int64_t)ap.n) - 1) / PA_KT + 1; };
    int64_t head_tiles = 0;
    for (int i = 0; i < nq; i++) head_tiles += tiles(i);
    const int64_t all = head_tiles * ap.nh, share = (all + G - 1) / G, waves = (total + G - 1) / G;
    // one by one: the idle places of the last round are at least the shortest item each
    const int64_t one_by_one = std::max(tiles(nq - 1), share + (waves * G - total) * tiles(0) / G);
    ap.shares = 0; ap.records = nullptr; ap.head_tiles = (int)head_tiles;
    if (one_by_one > share + (GQA ? (int64_t)PA_MERGE_TILES : std::max<int64_t>(PR_MERGE_TILES, share / 4)) && share >= 2 && all < (1LL << 31)) {
        const int s = cwk_reserve_scratch(ctx, (size_t)2 * H * G * PA_RECORD * sizeof(float));
        if (s != CWK_OK) return s;
        ap.shares = G; ap.records = ctx->scratch;
    }
    const int nflags = total + (ap.shares ? G : 0);
    ap.counter = ap.flags + nflags;
    CWK_CUDA(ctx, cudaMemsetAsync(ap.flags, 0, (size_t)(nflags + 3) * sizeof(int), ctx->stream));
    if (exact_only) {       // every item flagged (any non-zero word), the flag count non-zero, the two item counters back to zero
        CWK_CUDA(ctx, cudaMemsetAsync(ap.flags, 1, (size_t)(nflags + 3) * sizeof(int), ctx->stream));
        CWK_CUDA(ctx, cudaMemsetAsync(ap.counter, 0, 2 * sizeof(int), ctx->stream));
    }
    if (!exact_only) {
        CwkKernelTimer timer(ctx);
        const int grid = H * (ap.shares ? G : std::min(total, G));
        if constexpr (GQA) CWK_CUDA(ctx, cwk_launch_early(prefill_attn_kernel<4, CFG, GQA>, dim3(grid), dim3(PA_THREADS<4>), CFG::SMEM, ctx->stream, tm_k, tm_c, ap));
        else CWK_CUDA(ctx, cwk_launch_early(prefill_pair_kernel, dim3(grid), dim3(PR_THREADS), PrCfg<CFG>::SMEM, ctx->stream, tm_k, tm_c, ap));
        CWK_LAUNCH_CHECK(ctx, "prefill attention");
    }
    // the repair pass: items whose flag is clear are skipped
    CWK_CUDA(ctx, cwk_launch_early(prefill_attn_kernel<1, CFG, GQA>, dim3(ap.shares ? H * G : std::min(H * total, ctx->sm_count)), dim3(PA_THREADS<1>), CFG::SMEM, ctx->stream, tm_k, tm_c, ap));
    CWK_LAUNCH_CHECK(ctx, "prefill_attn_kernel<1>");
    if (ap.shares) {
        CWK_CUDA(ctx, cwk_launch_early(attn_merge_kernel<GQA>, dim3(ap.shares, PA_DV / PA_MC, H), dim3(128), 0, ctx->stream, ap));
        CWK_LAUNCH_CHECK(ctx, "attn_merge_kernel");
    }
    return CWK_OK;
}

// ---------------------------------------------------------------------------------------------------------------
// Key expansion: Kx[h][c][0:128] = W_uk[h] lat[c], Kx[h][c][128:192] = k_rope[c].
//
// Pairs of CTAs (M 256): each has 128 of a tile's 256 tokens and 64 of the head's 128 rows of W_uk, so that the weights take half the
// shared memory and the latent ring has four stages; with the whole of W_uk in one CTA there was room for two, 64 KB in
// flight per SM. What a tile waited for was its epilogue on four warps (3510 keys x 64 heads: 64 us, the stores 13, the MMAs
// 18): now eight, a half of the columns each.
constexpr int KX_TOK = 128, KX_NOPE = 128, KX_ST = 4;
constexpr int KX_W_BYTES = KX_NOPE / 2 * PA_L * 2;    // 65536: eight [64 d][64 l] blocks
constexpr int KX_A_BYTES = KX_TOK * 128 * 2;          // 32768: two [128 tok][64 l] blocks = one 128-wide chunk of the latent
constexpr int KX_OFF_W = 0, KX_OFF_A = KX_W_BYTES, KX_OFF_STG = KX_OFF_A + KX_ST * KX_A_BYTES, KX_OFF_BAR = KX_OFF_STG + 8 * 4096;
constexpr int KX_SMEM = KX_OFF_BAR + 256 + 1024, KX_THREADS = 384;
static_assert(KX_SMEM <= 232448, "shared-memory budget");
enum { KB_WFULL = 0, KB_AFULL = 1, KB_AEMPTY = KB_AFULL + KX_ST, KB_DFULL = KB_AEMPTY + KX_ST, KB_DEMPTY = KB_DFULL + 2, KB_COUNT = KB_DEMPTY + 2 };

struct KexpParams {
    const uint16_t *cache;    // bf16 [T][576]
    uint16_t *kx;             // bf16 [nh][T][192]: head-major, so that a head's key tile is one contiguous 24 KB
    int T, nh;
    int *err;
};

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(KX_THREADS, 1)
kexp_tc_kernel(const __grid_constant__ CUtensorMap tm_lat, const __grid_constant__ CUtensorMap tm_w, const KexpParams p) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t *sm = smem_raw + (base - raw);
    const uint32_t bar0 = base + KX_OFF_BAR;
    auto bar = [&](int i) { return bar0 + 8u * (uint32_t)i; };
    uint32_t *s_tmem = reinterpret_cast<uint32_t *>(sm + KX_OFF_BAR + 8 * KB_COUNT + 8);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int h = blockIdx.y, rank = (int)cluster_rank();
    const int pair = (int)blockIdx.x >> 1, pairs = (int)gridDim.x >> 1;
    const int ntiles = (p.T + 2 * KX_TOK - 1) / (2 * KX_TOK);
    const int nt = (ntiles - pair + pairs - 1) / pairs;                                  // tiles g, g + G, ...
    if (nt <= 0) return;
    const int nch = nt * 4;                                                              // 128-wide chunks of the 512 latent dims

    if (tid == 0) {
        asm volatile("prefetch.tensormap [%0];" ::"l"(&tm_lat) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&tm_w) : "memory");
        for (int i = 0; i < KB_COUNT; i++) mbar_init(bar(i), i >= KB_DEMPTY ? 16u : 1u);      // DEMPTY: the epilogue warps of both CTAs, at the first one's barrier
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    cwk_pdl_launch();
    cwk_pdl_wait();
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(s_tmem)), "r"(256u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();
    tc_fence_after();
    const uint32_t tmem = *s_tmem;

    if (warp == 0) {
        if (lane == 0) {
            if (rank == 0) mbar_expect_tx(bar(KB_WFULL), 2 * KX_W_BYTES);                // both CTAs' bytes are counted where the issuer waits
            tma_load_3d_pair(base + KX_OFF_W, &tm_w, 0, h * KX_NOPE + rank * (KX_NOPE / 2), 0, cluster_addr(bar(KB_WFULL), 0));
            bool ok = true;
            int issued = 0;
            for (int c = 0; c < nch && ok; c++) {
                const int slot = c % KX_ST, use = c / KX_ST;
                ok = mbar_wait(bar(KB_AEMPTY + slot), (uint32_t)((use & 1) ^ 1), p.err, 1101);
                if (!ok) break;
                const int tile = pair + (c >> 2) * pairs;
                if (rank == 0) mbar_expect_tx(bar(KB_AFULL + slot), 2 * KX_A_BYTES);
                tma_load_3d_pair(base + KX_OFF_A + slot * KX_A_BYTES, &tm_lat, 0, (tile * 2 + rank) * KX_TOK, (c & 3) * 2, cluster_addr(bar(KB_AFULL + slot), 0));
                issued = c + 1;
            }
            // the issuer commits to both CTAs: none of these arrivals may still be on its way here when this CTA leaves
            for (int c = max(0, nch - KX_ST); c < nch && ok; c++)
                ok = mbar_wait(bar(KB_AEMPTY + c % KX_ST), (uint32_t)((c / KX_ST) & 1), p.err, 1108);
            if (!ok && rank == 0) {
                mbar_wait(bar(KB_WFULL), 0, p.err, 1102);
                for (int c = (issued > KX_ST ? issued - KX_ST : 0); c < issued; c++) mbar_wait(bar(KB_AFULL + c % KX_ST), (uint32_t)((c / KX_ST) & 1), p.err, 1103);
            }
        }
    } else if (warp == 1) {
        if (lane == 0 && rank == 0) {
            constexpr uint32_t ID = idesc_bf16(2 * KX_TOK, KX_NOPE, 0, 0);
            const uint64_t dW = smem_desc(base + KX_OFF_W, 16, 1024);
            bool ok = mbar_wait(bar(KB_WFULL), 0, p.err, 1104);
            for (int c = 0; c < nch && ok; c++) {
                const int slot = c % KX_ST, use = c / KX_ST, ti = c >> 2, kc = c & 3, db = ti & 1;
                if (kc == 0) ok = mbar_wait(bar(KB_DEMPTY + db), (uint32_t)(((ti >> 1) & 1) ^ 1), p.err, 1105);
                if (ok) ok = mbar_wait(bar(KB_AFULL + slot), (uint32_t)(use & 1), p.err, 1106);
                if (!ok) break;
                tc_fence_after();
                const uint64_t dA = smem_desc(base + KX_OFF_A + slot * KX_A_BYTES, 16, 1024);
#pragma unroll
                for (int s = 0; s < 8; s++)       // chunk kc covers W blocks 2 kc and 2 kc + 1
                    umma_bf16_pair(tmem + db * KX_NOPE, dA + (uint64_t)(((s >> 2) * (KX_TOK * 128) + (s & 3) * 32) >> 4),
                                   dW + (uint64_t)((((kc * 2 + (s >> 2)) * (KX_NOPE / 2 * 128)) + (s & 3) * 32) >> 4), ID, (kc | s) != 0);
                umma_commit_pair(bar(KB_AEMPTY + slot));
                if (kc == 3) umma_commit_pair(bar(KB_DFULL + db));
            }
        }
    } else if (warp >= 4) {
        const int q4 = warp & 3, half = (warp - 4) >> 2;      // this warp's rows; its 64 columns, and half of the rows' rope tails
        const uint32_t tlane = tmem + ((uint32_t)(q4 * 32) << 16);
        uint8_t *stg = sm + KX_OFF_STG + (warp - 4) * 4096;
        bool ok = true;
        for (int ti = 0; ti < nt && ok; ti++) {
            const int db = ti & 1;
            const int t0w = ((pair + ti * pairs) * 2 + rank) * KX_TOK + q4 * 32;
            // rope tail first (independent of the MMAs): 128 bytes per token, eight lanes per row
#pragma unroll
            for (int r8 = 0; r8 < 4; r8++) {
                const int rr = (half * 4 + r8) * 4 + (lane >> 3), jj = lane & 7;
                if (t0w + rr < p.T) {
                    const uint4 w = *reinterpret_cast<const uint4 *>(p.cache + (int64_t)(t0w + rr) * PA_ROW + PA_L + jj * 8);
                    *reinterpret_cast<uint4 *>(p.kx + ((int64_t)h * p.T + t0w + rr) * PaMla::DQK + KX_NOPE + jj * 8) = w;
                }
            }
            ok = mbar_wait_warp(bar(KB_DFULL + db), (uint32_t)((ti >> 1) & 1), p.err, 1107);
            if (!ok) break;
            tc_fence_after();
            {
                const int c = half;
                uint32_t v[64];
                TMEM_LD16(v, 0, tlane + db * KX_NOPE + c * 64);
                TMEM_LD16(v, 16, tlane + db * KX_NOPE + c * 64 + 16);
                TMEM_LD16(v, 32, tlane + db * KX_NOPE + c * 64 + 32);
                TMEM_LD16(v, 48, tlane + db * KX_NOPE + c * 64 + 48);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    uint4 w;
                    w.x = pack_bf16x2(__uint_as_float(v[8 * j]), __uint_as_float(v[8 * j + 1]));
                    w.y = pack_bf16x2(__uint_as_float(v[8 * j + 2]), __uint_as_float(v[8 * j + 3]));
                    w.z = pack_bf16x2(__uint_as_float(v[8 * j + 4]), __uint_as_float(v[8 * j + 5]));
                    w.w = pack_bf16x2(__uint_as_float(v[8 * j + 6]), __uint_as_float(v[8 * j + 7]));
                    *reinterpret_cast<uint4 *>(stg + lane * 128 + ((j ^ (lane & 7)) << 4)) = w;
                }
                __syncwarp();
#pragma unroll
                for (int r8 = 0; r8 < 8; r8++) {
                    const int rr = r8 * 4 + (lane >> 3), jj = lane & 7;
                    const uint4 w = *reinterpret_cast<const uint4 *>(stg + rr * 128 + ((jj ^ (rr & 7)) << 4));
                    if (t0w + rr < p.T)
                        *reinterpret_cast<uint4 *>(p.kx + ((int64_t)h * p.T + t0w + rr) * PaMla::DQK + c * 64 + jj * 8) = w;
                }
                __syncwarp();
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(cluster_addr(bar(KB_DEMPTY + db), 0));
        }
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();                                          // the pair's barriers and tensor memory stay until both are done
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256u) : "memory");
    }
}

bool encode3(CUtensorMap *tm, const void *ptr, uint64_t rows, uint64_t blocks, uint64_t row_bytes, uint32_t box_rows, uint32_t box_blocks) {
    CwkEncodeTiledFn enc = cwk_encode_tiled_fn();
    if (!enc) return false;
    cuuint64_t dims[3] = {64, rows, blocks};
    cuuint64_t strides[2] = {row_bytes, 128};
    cuuint32_t box[3] = {64, box_rows, box_blocks};
    cuuint32_t es[3] = {1, 1, 1};
    return enc(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void *>(ptr), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

// Whether cwk_mla_prefill_attn_tc can take these operands (asked before the caller rotates Q in place).
bool cwk_mla_prefill_attn_tc_ok(const void *Q, const void *cache, const void *Wuk, const void *kx, const void *out) {
    if (!cwk_encode_tiled_fn()) return false;
    return ((reinterpret_cast<uintptr_t>(Q) | reinterpret_cast<uintptr_t>(cache) | reinterpret_cast<uintptr_t>(Wuk) | reinterpret_cast<uintptr_t>(kx) |
             reinterpret_cast<uintptr_t>(out)) & 15) == 0;
}

// Q bf16 [n][nh][192]; rot = (cos, sin) of the rope pairs at the queries' positions, f32 [n][32][2], 16-byte aligned (NULL: Q has been
// rotated); cache bf16 [pos0 + n][576] (latent | rope key);
// Wuk bf16 [nh][128][512]; kx = workspace bf16 [nh][pos0 + n][192]; flags = workspace int32, one per item of the
// attention (ceil(n / 128) x nh x 2) and per SM plus three counters; out bf16 [n][nh][512]. exact_only: skip the fast form and run
// the exact form on every item (for tests).
// Returns CWK_ERR_UNSUPPORTED (no error text) when the tensor path cannot run.
int cwk_mla_prefill_attn_tc(cwk_ctx *ctx, const void *Q, const float *rot, const void *cache, const void *Wuk, void *kx, int *flags, int64_t pos0, int n, int nh,
                            float scale, void *out, int exact_only) {
    if (!cwk_encode_tiled_fn()) return CWK_ERR_UNSUPPORTED;
    if ((reinterpret_cast<uintptr_t>(Q) | reinterpret_cast<uintptr_t>(cache) | reinterpret_cast<uintptr_t>(Wuk) | reinterpret_cast<uintptr_t>(kx) |
         reinterpret_cast<uintptr_t>(out)) & 15)
        return CWK_ERR_UNSUPPORTED;
    int s = cwk_ensure_err_word(ctx);
    if (s != CWK_OK) return s;
    const int T = (int)(pos0 + n);
    CUtensorMap tm_lat, tm_w, tm_k, tm_c;
    if (!encode3(&tm_lat, cache, (uint64_t)T, PA_L / 64, PA_ROW * 2, KX_TOK, 2) ||                 // latent dims only: block index 8 (rope) stays out
        !encode3(&tm_w, Wuk, (uint64_t)nh * KX_NOPE, PA_L / 64, PA_L * 2, KX_NOPE / 2, PA_L / 64) ||
        !encode3(&tm_k, kx, (uint64_t)nh * T, 3, PaMla::DQK * 2, PA_KT, 3) ||            // rows past a head's last key belong to the next head: every such key is masked

        !encode3(&tm_c, cache, (uint64_t)T, PA_L / 64, PA_ROW * 2, PA_KT, 4))
        return cwk_fail(ctx, CWK_ERR_CUDA, "cuTensorMapEncodeTiled failed for the prefill attention operands");
    static bool attr_set[16] = {false};
    if (!attr_set[ctx->device & 15]) {
        CWK_CUDA(ctx, cudaFuncSetAttribute(kexp_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, KX_SMEM));
        attr_set[ctx->device & 15] = true;
    }
    {
        KexpParams kp;
        kp.cache = (const uint16_t *)cache; kp.kx = (uint16_t *)kx; kp.T = T; kp.nh = nh; kp.err = ctx->dev_err;
        const int ntiles = (T + 2 * KX_TOK - 1) / (2 * KX_TOK);
        const int G = std::max(1, std::min(ntiles, ctx->sm_count / 2 / std::max(1, nh)));      // pairs per head
        CwkKernelTimer timer(ctx);
        CWK_CUDA(ctx, cwk_launch_early(kexp_tc_kernel, dim3(2 * G, nh), dim3(KX_THREADS), KX_SMEM, ctx->stream, tm_lat, tm_w, kp));
        CWK_LAUNCH_CHECK(ctx, "kexp_tc_kernel");
    }
    AttnParams ap{};
    ap.q = (const uint16_t *)Q; ap.rot = (const float4 *)rot; ap.out = (uint16_t *)out; ap.n = n; ap.nh = nh; ap.T = T; ap.pos0 = pos0; ap.group = 1;
    ap.scale_log2 = scale * 1.4426950408889634f; ap.flags = flags; ap.err = ctx->dev_err;
    return attn_launch<PaMla, false>(ctx, ap, tm_k, tm_c, exact_only);
}

// Causal GQA prefill on the same kernel (Qwen3.5 full-attention layers, src/q35_model.c:1713-1746): per query head,
// 128 consecutive queries are the MMA's rows; keys and values are the 256-wide rows of the head's KV head, streamed in
// 64-key tiles by TMA straight from the caches. Q bf16 [n][nh][256]; K, V bf16 [pos + n][nkv][256]; out bf16
// [n][nh][256]; flags = workspace int32 [ceil(n / 128) * nh + number of SMs + 3]. Returns CWK_ERR_UNSUPPORTED (no error text) when the
// tensor path cannot take the operands.
int cwk_gqa_prefill_tc(cwk_ctx *ctx, const void *Q, const void *K, const void *V, int64_t pos, int n, int nh, int nkv, int hd,
                       float scale, void *out, int *flags) {
    if (!cwk_encode_tiled_fn() || hd != 256 || nkv <= 0 || nh % nkv) return CWK_ERR_UNSUPPORTED;
    if ((reinterpret_cast<uintptr_t>(Q) | reinterpret_cast<uintptr_t>(K) | reinterpret_cast<uintptr_t>(V) | reinterpret_cast<uintptr_t>(out)) & 15)
        return CWK_ERR_UNSUPPORTED;
    int s = cwk_ensure_err_word(ctx);
    if (s != CWK_OK) return s;
    const int T = (int)(pos + n);
    CUtensorMap tm_k, tm_v;
    // the caches as [64][rows][nkv * 4 column blocks]: a tile is one box of 64 keys x the 4 blocks of one KV head
    if (!encode3(&tm_k, K, (uint64_t)T, (uint64_t)nkv * 4, (uint64_t)nkv * hd * 2, PA_KT, 4) ||
        !encode3(&tm_v, V, (uint64_t)T, (uint64_t)nkv * 4, (uint64_t)nkv * hd * 2, PA_KT, 4))
        return cwk_fail(ctx, CWK_ERR_CUDA, "cuTensorMapEncodeTiled failed for the GQA prefill operands");
    AttnParams ap{};
    ap.q = (const uint16_t *)Q; ap.out = (uint16_t *)out; ap.n = n; ap.nh = nh; ap.T = T; ap.pos0 = pos; ap.group = nh / nkv;
    ap.scale_log2 = scale * 1.4426950408889634f; ap.flags = flags; ap.err = ctx->dev_err;
    return attn_launch<PaGqa, true>(ctx, ap, tm_k, tm_v, 0);
}
