// gqa_decode.cu -- Qwen3.5-style GQA single-query decode (dec_scores / dec_softmax / dec_out_slices and the slice sum,
// src/q35_model.c:1460-1518, :1656-1712) for a batch of sequences with lengths of their own.
//
// Four FLOP per cached byte: the kernel's whole job is to keep copies in flight. So no warp ever waits for another one:
// every warp has a ring of its own (three stages of sixteen keys, K and V, filled by asynchronous copies two stages ahead),
// its own running maximum, sum and output, and writes its own record; what a tile costs in latency -- a chain of sixteen
// score MMAs, the exponentials, sixteen value MMAs -- is hidden behind the two other stages and the three other warps.
// (With a block's eight warps sharing each 64-key tile and meeting at barriers, as the kernel for prompts does, that chain
// was 4.4 k cycles per tile, against 2.8 k that the tile's bytes take at an SM's share of HBM.)
//
// Both products are issued transposed, with the keys or the value columns as the sixteen rows of mma.m16n8k16 and the
// query heads of one KV head (at most eight) as its eight columns: half the MMAs of the form with heads as rows padded to
// sixteen, half the accumulators (64 registers for 256 columns), the query in registers, and a warp's probabilities turn from
// result into operand with two 8 x 8 transposes.
//
// The steps of all sequences (sixteen keys of up to four KV heads, one per warp: their rows are neighbours in memory) are
// dealt out in equal contiguous ranges, one per SM, worked out from the lengths on the device: every SM has the same
// number of bytes to read, and a block goes from one sequence to the next without its ring running dry.
#include <algorithm>

#include "cwk_common.cuh"

namespace {

constexpr int GW = 4;                 // warps per block
constexpr int GK = 16;                // keys per warp and step
constexpr float GQ_LAZY = 8.f;        // a score may outrun the reference exponent by 2^8 before a rescale

struct GqaDecodeParams {
    const uint16_t *q, *k, *v;        // q bf16 [B][nh][hd]; caches: sequence b at + b * seq_stride, rows of ld
    int64_t seq_stride, ld;
    const int32_t *kv_len, *sel;      // [B]; optional row lists [B][sel_ld]
    int64_t sel_ld;
    int B, nh, nkv, group, hb;        // hb: KV heads a block works on at once (4, 2 or 1)
    float scale_log2;
    float *rec;                       // [slot][warp][group][hd + 2]
    int2 *meta;                       // [B][nkv / hb]: first slot, number of slots
};

// A block's place in the list of all steps: sequence, group of KV heads, step within it.
struct GqaPlace {
    int b, hg, step, steps, len;      // steps: of this sequence (and head group)
};
__device__ __forceinline__ int steps_of(const GqaDecodeParams &p, int b) { return b < p.B ? (max(p.kv_len[b], 0) + GK * (GW / p.hb) - 1) / (GK * (GW / p.hb)) : 0; }

// This block's range [lo, hi) of all steps, and where it begins. Every warp works it out for itself; the first one notes, for
// every (sequence, head group) whose first step is in the range, its first record slot (slots are numbered by head group
// plus block: one of the two grows from record to record) and their number.
__device__ __forceinline__ int gqa_range(const GqaDecodeParams &p, int lane, bool note, GqaPlace &at) {
    const int nhg = p.nkv / p.hb;
    int64_t total = 0;
    for (int b0 = 0; b0 < p.B; b0 += 32) {
        int v = steps_of(p, b0 + lane);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        total += v;
    }
    total *= nhg;
    const int64_t G = max((int64_t)1, min((int64_t)gridDim.x, total)), g = blockIdx.x;      // no block between two others is left without a step
    const int64_t lo = g < G ? total * g / G : total, hi = g < G ? total * (g + 1) / G : total;
    int64_t before = 0;
    for (int b0 = 0; b0 < p.B; b0 += 32) {
        const int mine = steps_of(p, b0 + lane);
        int v = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += u;
        }
        const int64_t s0 = (before + v - mine) * nhg, s1 = s0 + (int64_t)mine * nhg;       // this lane's sequence: steps [s0, s1)
        const bool here = mine > 0 && s0 <= lo && lo < s1 && lo < hi;
        const uint32_t who = __ballot_sync(0xffffffffu, here);
        if (who) {
            const int src = __ffs(who) - 1;
            at.b = b0 + src;
            at.steps = __shfl_sync(0xffffffffu, mine, src);
            const int off = (int)__shfl_sync(0xffffffffu, (int)(lo - s0), src);
            at.hg = off / at.steps;
            at.step = off % at.steps;
        }
        if (note && b0 + lane < p.B) {
            if (mine == 0) {
                if (s0 > 0 ? (lo < s0 && s0 <= hi) : g == 0)
                    for (int h = 0; h < nhg; h++) p.meta[(b0 + lane) * nhg + h] = make_int2(0, 0);
            } else if (s0 < hi && s1 > lo) {
                const int64_t h0 = lo > s0 ? (lo - s0 + mine - 1) / mine : 0;              // first head group that begins here
                for (int64_t h = h0; h < nhg && s0 + h * mine < hi; h++) {
                    const int64_t g1 = ((s0 + (h + 1) * mine) * G - 1) / total;              // the block with its last step
                    p.meta[(b0 + lane) * nhg + h] = make_int2((int)((b0 + lane) * nhg + h + g), (int)(g1 - g + 1));
                }
            }
        }
        before += __shfl_sync(0xffffffffu, v, 31);
    }
    return (int)(hi - lo);
}
__device__ __forceinline__ void gqa_advance(const GqaDecodeParams &p, GqaPlace &at) {      // to the next step; there is one
    if (++at.step < at.steps) return;
    at.step = 0;
    if (++at.hg < p.nkv / p.hb) return;
    at.hg = 0;
    do {
        at.b++;
        at.len = p.kv_len[at.b];
    } while (at.len <= 0);
    at.steps = steps_of(p, at.b);
}

template <int HD>
__global__ void __launch_bounds__(32 * GW) gqa_decode_kernel(const GqaDecodeParams p) {
    constexpr int CH = HD / 8;                            // 16-byte pieces per row
    constexpr int STAGES = HD == 256 ? 3 : 6;
    constexpr int KB = GK * HD * 2;                       // bytes of a stage's K (and of its V)
    extern __shared__ __align__(128) uint8_t smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, lg = lane >> 2, lt = lane & 3;
    const uint32_t ring = smem_u32(smem) + warp * STAGES * 2 * KB;
    const int sub = warp / p.hb, wh = warp % p.hb;        // which sixteen keys of a step, which KV head of the group
    const int keys = GK * (GW / p.hb);
    GqaPlace at{0, 0, 0, 0, 0};
    cwk_pdl_launch();
    cwk_pdl_wait();
    const int n = gqa_range(p, lane, warp == 0, at);
    if (n <= 0) return;
    at.len = p.kv_len[at.b];
    GqaPlace ld = at;                                     // the step being loaded
    auto load = [&](int slot) {
        const int j0 = ld.step * keys + sub * GK, kvh = ld.hg * p.hb + wh;
        const uint16_t *kb = p.k + (int64_t)ld.b * p.seq_stride + kvh * HD, *vb = p.v + (int64_t)ld.b * p.seq_stride + kvh * HD;
        int row = j0 + (lane & 15);
        if (p.sel) row = row < ld.len ? p.sel[(int64_t)ld.b * p.sel_ld + row] : 0;
        const uint32_t dst = ring + slot * 2 * KB;
        constexpr int RPI = 32 / CH;                      // rows per instruction: 1 or 2
        const int c = lane % CH, rr = lane / CH;
#pragma unroll
        for (int i = 0; i < GK / RPI; i++) {
            const int r = i * RPI + rr;
            const bool ok = j0 + r < ld.len;
            const int64_t off = (int64_t)__shfl_sync(0xffffffffu, row, r) * p.ld + c * 8;
            const uint32_t d = dst + r * HD * 2 + ((c ^ (r & 7)) << 4);
            cp_async16(d, kb + (ok ? off : 0), ok);
            cp_async16(d + KB, vb + (ok ? off : 0), ok);
        }
    };
    for (int s = 0; s < STAGES - 1; s++) {
        if (s < n) {
            load(s);
            if (s + 1 < n) gqa_advance(p, ld);
        }
        cp_async_commit();
    }
    uint32_t bq[HD / 16][2];                              // the query heads, as the score MMAs' second operand
    float acc[HD / 16][4];                                // value columns 16 i + lg (+ 8) of heads 2 lt, 2 lt + 1
    float m0 = 0.f, m1 = 0.f, l0 = 0.f, l1 = 0.f;
    bool fresh = true;
    for (int s = 0; s < n; s++) {
        if (fresh) {
            const uint16_t *qr = p.q + ((int64_t)at.b * p.nh + (at.hg * p.hb + wh) * p.group + lg) * HD;
#pragma unroll
            for (int i = 0; i < HD / 16; i++) {
                bq[i][0] = lg < p.group ? *reinterpret_cast<const uint32_t *>(qr + i * 16 + 2 * lt) : 0u;
                bq[i][1] = lg < p.group ? *reinterpret_cast<const uint32_t *>(qr + i * 16 + 8 + 2 * lt) : 0u;
                acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
            }
            l0 = l1 = 0.f;
        }
        cp_async_wait<STAGES - 2>();
        __syncwarp();                                     // every lane's copies of this step have landed; the last step's slot has been read
        if (s + STAGES - 1 < n) {
            load((s + STAGES - 1) % STAGES);
            if (s + STAGES < n) gqa_advance(p, ld);
        }
        cp_async_commit();
        const uint32_t tK = ring + (s % STAGES) * 2 * KB, tV = tK + KB;
        float c0[4] = {0.f, 0.f, 0.f, 0.f}, c1[4] = {0.f, 0.f, 0.f, 0.f};      // two chains
        {
            const uint32_t ra = tK + (lane & 15) * HD * 2;
            const int x = lane & 7, h = lane >> 4;
#pragma unroll
            for (int i = 0; i < HD / 16; i++) {
                uint32_t a[4];
                ldmatrix_x4(a[0], a[1], a[2], a[3], ra + (((2 * i + h) ^ x) << 4));
                mma_bf16_16816((i & 1) ? c1 : c0, a, bq[i][0], bq[i][1]);
            }
        }
        const int ja = at.step * keys + sub * GK + lg;    // this lane's keys: ja and ja + 8
        const bool va = ja < at.len, vb = ja + 8 < at.len;
        const float s0 = va ? (c0[0] + c1[0]) * p.scale_log2 : -INFINITY, s1 = va ? (c0[1] + c1[1]) * p.scale_log2 : -INFINITY;
        const float s2 = vb ? (c0[2] + c1[2]) * p.scale_log2 : -INFINITY, s3 = vb ? (c0[3] + c1[3]) * p.scale_log2 : -INFINITY;
        float x0 = fmaxf(s0, s2), x1 = fmaxf(s1, s3);
        if (fresh || __any_sync(0xffffffffu, x0 > m0 + GQ_LAZY || x1 > m1 + GQ_LAZY)) {
#pragma unroll
            for (int o = 4; o < 32; o <<= 1) {
                x0 = fmaxf(x0, __shfl_xor_sync(0xffffffffu, x0, o));
                x1 = fmaxf(x1, __shfl_xor_sync(0xffffffffu, x1, o));
            }
            if (fresh) {                                  // (no key at all in this warp's share: any exponent will do)
                m0 = x0 == -INFINITY ? 0.f : x0;
                m1 = x1 == -INFINITY ? 0.f : x1;
            } else {
                const float n0 = fmaxf(m0, x0), n1 = fmaxf(m1, x1), a0 = exp2f(m0 - n0), a1 = exp2f(m1 - n1);
                m0 = n0; m1 = n1; l0 *= a0; l1 *= a1;
#pragma unroll
                for (int i = 0; i < HD / 16; i++) { acc[i][0] *= a0; acc[i][1] *= a1; acc[i][2] *= a0; acc[i][3] *= a1; }
            }
        }
        const float p0 = exp2f(s0 - m0), p1 = exp2f(s1 - m1), p2 = exp2f(s2 - m0), p3 = exp2f(s3 - m1);
        l0 += p0 + p2;
        l1 += p1 + p3;
        uint32_t b0 = pack_bf16x2(p0, p1), b1 = pack_bf16x2(p2, p3);             // [8 keys][8 heads] each -> [8 heads][8 keys]
        asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %0;" : "+r"(b0));
        asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %0;" : "+r"(b1));
        {
            const int key = (lane & 7) + ((lane >> 4) << 3), h = (lane >> 3) & 1, x = lane & 7;
            const uint32_t ra = tV + key * HD * 2;
#pragma unroll
            for (int i = 0; i < HD / 16; i++) {
                uint32_t a[4];
                ldmatrix_x4_trans(a[0], a[1], a[2], a[3], ra + (((2 * i + h) ^ x) << 4));
                mma_bf16_16816(acc[i], a, b0, b1);
            }
        }
        fresh = at.step + 1 == at.steps;
        if (fresh || s + 1 == n) {                        // the end of what this block has of the sequence's head group: its record
#pragma unroll
            for (int o = 4; o < 32; o <<= 1) {
                l0 += __shfl_xor_sync(0xffffffffu, l0, o);
                l1 += __shfl_xor_sync(0xffffffffu, l1, o);
            }
            const int64_t slot = (int64_t)at.b * (p.nkv / p.hb) + at.hg + blockIdx.x;
            float *r = p.rec + (slot * GW + warp) * p.group * (HD + 2);
            const int h0 = 2 * lt;
            if (lg == 0) {
                if (h0 < p.group) { r[h0 * (HD + 2)] = l0 > 0.f ? m0 : -INFINITY; r[h0 * (HD + 2) + 1] = l0; }
                if (h0 + 1 < p.group) { r[(h0 + 1) * (HD + 2)] = l1 > 0.f ? m1 : -INFINITY; r[(h0 + 1) * (HD + 2) + 1] = l1; }
            }
#pragma unroll
            for (int i = 0; i < HD / 16; i++) {
                float *o = r + 2 + i * 16 + lg;
                if (h0 < p.group) { o[h0 * (HD + 2)] = acc[i][0]; o[h0 * (HD + 2) + 8] = acc[i][2]; }
                if (h0 + 1 < p.group) { o[(h0 + 1) * (HD + 2)] = acc[i][1]; o[(h0 + 1) * (HD + 2) + 8] = acc[i][3]; }
            }
        }
        if (s + 1 < n) gqa_advance(p, at);
    }
    cp_async_wait<0>();
}

// grid (query head, sequence), (HD / 2) x GROUPS threads: two columns each, the records of the head's blocks and warps dealt
// out to the groups (one sequence has a record from every block: 148 in a row are 20 us of loads for one group of threads).
template <int HD, int GROUPS>
__global__ void __launch_bounds__(HD / 2 * GROUPS) gqa_merge_kernel(const GqaDecodeParams p, uint16_t *out) {
    constexpr int NT = HD / 2;
    __shared__ float s_m[GROUPS], s_l[GROUPS];
    __shared__ float2 s_o[GROUPS][NT];
    const int h = blockIdx.x, b = blockIdx.y, kvh = h / p.group, nhg = p.nkv / p.hb, ks = GW / p.hb;
    const int g = threadIdx.x / NT, tid = threadIdx.x % NT;
    cwk_pdl_launch();
    cwk_pdl_wait();
    const int2 meta = p.meta[b * nhg + kvh / p.hb];
    const int64_t rsz = (int64_t)p.group * (HD + 2);
    // record i: slot first + i / ks, warp (i % ks) * hb + kvh % hb
    const float *base = p.rec + ((int64_t)meta.x * GW + kvh % p.hb) * rsz + (int64_t)(h % p.group) * (HD + 2);
    const int cnt = meta.y * ks;
    auto at = [&](int i) { return base + (ks == 1 ? (int64_t)i * GW : (int64_t)(i / ks) * GW + (i % ks) * p.hb) * rsz; };
    float M = -INFINITY, den = 0.f, x = 0.f, y = 0.f;
    for (int i0 = g; i0 < cnt; i0 += 8 * GROUPS) {         // eight records' loads at once; the running maximum as the scores'
        float m[8], l[8];
        float2 o[8];
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const int i = i0 + j * GROUPS;
            const float *r = at(min(i, cnt - 1));
            m[j] = i < cnt ? r[0] : -INFINITY;
            l[j] = r[1];
            o[j] = *reinterpret_cast<const float2 *>(r + 2 + 2 * tid);
        }
        float mx = M;
#pragma unroll
        for (int j = 0; j < 8; j++) mx = fmaxf(mx, m[j]);
        if (mx == -INFINITY) continue;
        const float a = exp2f(M - mx);
        den *= a; x *= a; y *= a;
        M = mx;
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const float w = exp2f(m[j] - M);
            den += w * l[j]; x += w * o[j].x; y += w * o[j].y;
        }
    }
    if (GROUPS > 1) {
        if (tid == 0) { s_m[g] = M; s_l[g] = den; }
        s_o[g][tid] = make_float2(x, y);
        __syncthreads();
        if (g > 0) return;
        float mx = -INFINITY;
#pragma unroll
        for (int j = 0; j < GROUPS; j++) mx = fmaxf(mx, s_m[j]);
        den = x = y = 0.f;
#pragma unroll
        for (int j = 0; j < GROUPS; j++) {
            const float w = s_m[j] == -INFINITY ? 0.f : exp2f(s_m[j] - mx);
            den += w * s_l[j]; x += w * s_o[j][tid].x; y += w * s_o[j][tid].y;
        }
    }
    const float inv = den > 0.f ? 1.f / den : 0.f;
    *reinterpret_cast<uint32_t *>(out + ((int64_t)b * p.nh + h) * HD + 2 * tid) = pack_bf16x2(x * inv, y * inv);
}

template <int HD>
int launch(cwk_ctx *ctx, const GqaDecodeParams &p, int blocks, void *out) {
    constexpr int SMEM = GW * (HD == 256 ? 3 : 6) * 2 * GK * HD * 2;      // 192 KB
    static bool attr_set[16] = {false};
    if (!attr_set[ctx->device & 15]) {
        CWK_CUDA(ctx, cudaFuncSetAttribute(gqa_decode_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM));
        attr_set[ctx->device & 15] = true;
    }
    {
        CwkKernelTimer timer(ctx);
        CWK_CUDA(ctx, cwk_launch_early(gqa_decode_kernel<HD>, dim3(blocks), dim3(32 * GW), SMEM, ctx->stream, p));
        ctx->launches++;
    }
    const bool many = (int64_t)blocks * (GW / p.hb) * (p.nkv / p.hb) > 8 * (int64_t)p.B * (p.nkv / p.hb);      // records per head and sequence
    CWK_CUDA(ctx, cwk_launch_early(many ? gqa_merge_kernel<HD, 8> : gqa_merge_kernel<HD, 1>, dim3(p.nh, p.B), dim3(HD / 2 * (many ? 8 : 1)), 0, ctx->stream, p, (uint16_t *)out));
    ctx->launches++;
    return CWK_OK;
}

}  // namespace

// At most eight query heads per KV head (the caller checks everything else). max_blocks <= 0: one block per SM.
int cwk_gqa_decode_streams(cwk_ctx *ctx, const void *q, const void *K, const void *V, int64_t seq_stride, const int32_t *kv_len, int max_kv_len,
                           const int32_t *sel, int64_t sel_ld, int B, int nh, int nkv, int hd, float scale, void *out, int max_blocks) {
    GqaDecodeParams p;
    p.q = (const uint16_t *)q; p.k = (const uint16_t *)K; p.v = (const uint16_t *)V; p.seq_stride = seq_stride; p.ld = (int64_t)nkv * hd;
    p.kv_len = kv_len; p.sel = sel; p.sel_ld = sel_ld; p.B = B; p.nh = nh; p.nkv = nkv; p.group = nh / nkv;
    p.hb = nkv % 4 == 0 ? 4 : nkv % 2 == 0 ? 2 : 1;
    p.scale_log2 = scale * 1.4426950408889634f;
    // as many blocks as there can be steps, at most one per SM
    const int keys = GK * (GW / p.hb);
    const int64_t most = std::max<int64_t>(1, (int64_t)B * (nkv / p.hb) * ((max_kv_len + keys - 1) / keys));
    const int blocks = (int)std::min<int64_t>(most, max_blocks > 0 ? std::min(max_blocks, ctx->sm_count) : ctx->sm_count);
    const int64_t slots = (int64_t)B * (nkv / p.hb) + blocks;
    const size_t rec_bytes = (size_t)slots * GW * p.group * (hd + 2) * sizeof(float);
    int s = cwk_reserve_scratch(ctx, rec_bytes + (size_t)B * (nkv / p.hb) * sizeof(int2));
    if (s != CWK_OK) return s;
    p.rec = ctx->scratch;
    p.meta = (int2 *)((uint8_t *)ctx->scratch + rec_bytes);
    return hd == 256 ? launch<256>(ctx, p, blocks, out) : launch<128>(ctx, p, blocks, out);
}
