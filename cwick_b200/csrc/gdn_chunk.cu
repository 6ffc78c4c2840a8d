// gdn_chunk.cu -- the Gated DeltaNet scan of a PROMPT, chunk-parallel (head dims 128 x 128).
//
// lin_rec_heads (src/q35_model.c:1177-1264) walks the positions one after the other: per position and value
// head, S <- d S;  u = beta (v - S k);  S <- S + u k^T;  o = S q.  gdn.cu does the same, which is the right form
// for a decode step and the wrong one for a prompt: 4096 positions x two dependent 128-term sums each is
// 14 ms per layer on 32 of the 148 SMs. The recurrence is linear in S, so 64 positions can be taken at once:
// with G_t the running sum of log d inside the chunk and r(t, s) = exp(G_t - G_s),
//
//   A[t][s] = beta_t r(t, s) (k_t . k_s)  (s < t),      T = (I + A)^-1          (64 x 64, unit lower triangular)
//   W = T diag(beta e^G) K,    U~ = T diag(beta) V,     M[t][s] = r(t, s) (q_t . k_s)  (s <= t)
//
// depend on the chunk's inputs only (prep: every chunk of every head at the same time), and then per chunk,
// in order, with S0 the state at the chunk's start,
//
//   U = U~ - W S0^T,        S0^T <- e^(G_64) S0^T + K^T diag(e^(G_64 - G)) U
//
// (scan: the only serial part; a value row of S never meets another one, so one block per (head, 32 value columns))
// and last, again for every chunk at the same time, O = diag(e^G) Q S0^T + M U and the gated RMS norm of its rows
// (output). The scan leaves every chunk's S0 and U behind for it.
//
// Bound: 9.6 G multiply-adds for 4096 positions of 32 heads, in f32. On CUDA cores an SM does 128 of them a clock and
// loads 32 floats, so a tile of outputs has to be 8 x 8 per thread before the loads stop being the limit, and these
// products are too small for that (the three kernels that way, 4 x 4 per thread with paired fmas: 176 + 364 + 219 us).
// They run on the tensor cores instead, mma.sync with TF32 operands, at f32 precision: an operand x is the sum of two
// TF32 numbers, a product is hi hi + hi lo + lo hi, and sums longer than 64 terms are carried on in f32 registers, so that
// the tensor core's truncating adder only ever adds a few terms; against float64 the results are as close as those of f32
// multiply-adds (4.6e-7 relative, 4.4e-7 before). 475 TF32 multiply-adds a clock and SM (measured) / 3 = 158; tcgen05 would
// do four times that, but the scan's blocks are 32 columns wide and its chain of two products per chunk is latency.
// What is left is instructions around the MMAs: the split of the operands (two per float) and addresses, which is why the
// operands' places are worked out once per kernel and read sixteen bytes at a time where the contraction runs along rows
// (the order of its terms is free, so a thread's four consecutive floats serve two MMAs).
// 4096 positions x 32 heads: prep 457 -> 185 us, scan 856 -> 240 us, output with the norm in it (the norm alone took 97) 172 us.
//
// Results agree with the reference to rounding (a few 1e-7 relative), not bit for bit: the sums run in another order.
// The position-serial kernel stays the form for decode steps and short calls. A call's last, partial chunk is filled up
// with positions that change nothing (no decay, no write).
#include <algorithm>

#include "cwk_common.cuh"

namespace {

constexpr int GC = 64;            // positions per chunk
constexpr int GD = 128;           // head_k = head_v
constexpr int GJ = 32;            // value columns per scan block

__device__ __forceinline__ float gc_exp(float x) { return (float)exp((double)x); }

// x as two TF32 numbers: the MMA reads the upper 19 bits of an operand, so x itself serves as its own truncation and the
// second number is the rest.
__device__ __forceinline__ void split_tf32(float x, uint32_t &hi, uint32_t &lo) {
    hi = __float_as_uint(x);
    lo = __float_as_uint(x - __uint_as_float(hi & 0xffffe000u));
}
__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
// Operands of a step of 16 terms (two MMAs of 8), split. A: 16 rows, this lane's rows g = lane / 4 and g + 8; B: 8 columns,
// this lane's column g. Term order: the lane t = lane % 4 of a row holds terms 4t .. 4t + 3; the first MMA takes 4t and 4t + 1,
// the second 4t + 2 and 4t + 3, in A and B alike.
struct OpA { uint32_t hi[2][4], lo[2][4]; };
struct OpB { uint32_t hi[2][2], lo[2][2]; };
__device__ __forceinline__ OpA op_a(const float (&r0)[4], const float (&r1)[4]) {
    OpA o;
#pragma unroll
    for (int m = 0; m < 2; m++)
#pragma unroll
        for (int k = 0; k < 2; k++) {
            split_tf32(r0[2 * m + k], o.hi[m][2 * k], o.lo[m][2 * k]);
            split_tf32(r1[2 * m + k], o.hi[m][2 * k + 1], o.lo[m][2 * k + 1]);
        }
    return o;
}
__device__ __forceinline__ OpB op_b(const float (&c)[4]) {
    OpB o;
#pragma unroll
    for (int m = 0; m < 2; m++)
#pragma unroll
        for (int k = 0; k < 2; k++) split_tf32(c[2 * m + k], o.hi[m][k], o.lo[m][k]);
    return o;
}
// A sum in two parts: the products of the rounded operands, and those with a remainder.
struct Acc {
    float d[4], e[4];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int i = 0; i < 4; i++) d[i] = e[i] = 0.f;
    }
    __device__ __forceinline__ float sum(int i) const { return d[i] + e[i]; }
};
__device__ __forceinline__ void mma3(Acc &c, const OpA &a, const OpB &b) {
#pragma unroll
    for (int m = 0; m < 2; m++) {
        mma_tf32(c.e, a.hi[m], b.lo[m]);
        mma_tf32(c.d, a.hi[m], b.hi[m]);
        mma_tf32(c.e, a.lo[m], b.hi[m]);
    }
}
__device__ __forceinline__ void cp16(float *dst, const float *src, bool valid) { cp_async16(smem_u32(dst), src, valid); }

struct GdnChunkParams {
    const float *up, *gdec, *beta, *gate, *a_log, *dt_bias, *norm;
    float *S, *out;
    float *ws;                    // per (slot, head, chunk): W [64][128] | U~, then U, transposed [128][64] | M [64][64] | S0 [128 value][128 key] | G [64], its remainders [64]
    int n;                        // positions per slot
    int left;                     // positions of a slot from the segment's first on (the arrays begin there)
    int nchunks, nh, kv_group;    // chunks of the segment
    float rms_eps;
};
constexpr int WS_U = GC * GD, WS_M = 2 * GC * GD, WS_S = WS_M + GC * GC, WS_G = WS_S + GD * GD;
constexpr int64_t WS_PER = WS_G + 2 * GC;
// Bytes of workspace in use at a time. A cut costs the ends of three kernels, most of it the last, half-empty wave of the
// prep kernel: 4096 positions x 32 heads (303 MB) 573 us whole, 607 in two segments, 669 in four; 16384 positions 2207 whole
// (1.2 GB), 2286 in four segments. So a prompt of that common size stays whole, and longer ones stay within its bound.
constexpr int64_t WS_MAX = 320 << 20;

__device__ __forceinline__ float *ws_of(const GdnChunkParams &p, int b, int vh, int c) {
    return p.ws + (((int64_t)b * p.nh + vh) * p.nchunks + c) * WS_PER;
}
// Offset of the four floats `q` (entries 4q .. 4q + 3) of row r in a tile of WIDTH-wide rows. The pieces of a row are
// permuted so that (1) rows 2m and 2m + 1 keep four neighbouring pieces in different halves of the banks -- a 16-byte read of
// two rows by eight lanes -- and (2) rows r, r + 4, r + 8, r + 12 keep two neighbouring pieces in different quarters -- a word
// read of four rows by eight lanes each.
template <int WIDTH> __device__ __forceinline__ int piece(int r, int q) {
    const int x = ((r >> 1) & 1) | (((r >> 2) & 1) << 1) | (((r ^ (r >> 3)) & 1) << 2);
    return r * WIDTH + ((q ^ x) << 2);
}
// Where a lane finds its terms 16 kk + 4t .. + 3 of row r: the permutation swaps neighbouring steps or does not, so two
// pointers and a constant per pair of steps.
struct RowPtr { const float *p[2]; };
template <int WIDTH> __device__ __forceinline__ RowPtr row_ptr(const float *s, int r, int t) {
    return RowPtr{{s + piece<WIDTH>(r, t), s + piece<WIDTH>(r, 4 + t)}};
}
__device__ __forceinline__ void row4(float (&v)[4], const RowPtr &r, int kk) {
    const float4 f = *reinterpret_cast<const float4 *>(r.p[kk & 1] + (kk >> 1) * 32);
    v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
}
// The same terms of column c, where the terms are rows: rows 16 kk + 4t + e, whose permutation does not depend on kk.
struct ColPtr { const float *p[4]; };
template <int WIDTH> __device__ __forceinline__ ColPtr col_ptr(const float *s, int c, int t) {
    ColPtr o;
#pragma unroll
    for (int e = 0; e < 4; e++) o.p[e] = s + piece<WIDTH>(4 * t + e, c >> 2) + (c & 3);
    return o;
}
template <int WIDTH> __device__ __forceinline__ void col4(float (&v)[4], const ColPtr &c, int kk) {
#pragma unroll
    for (int e = 0; e < 4; e++) v[e] = c.p[e][kk * 16 * WIDTH];
}
struct RowPtrA { RowPtr r0, r1; };
template <int WIDTH> __device__ __forceinline__ RowPtrA row_ptr_a(const float *s, int r, int t) { return RowPtrA{row_ptr<WIDTH>(s, r, t), row_ptr<WIDTH>(s, r + 8, t)}; }
__device__ __forceinline__ OpA op_a(const RowPtrA &r, int kk) {
    float a[4], b[4];
    row4(a, r.r0, kk);
    row4(b, r.r1, kk);
    return op_a(a, b);
}
__device__ __forceinline__ OpB op_b(const RowPtr &r, int kk) {
    float a[4];
    row4(a, r, kk);
    return op_b(a);
}

// ---- prep: grid (chunk, key head, slot), 256 threads, the key head's value heads one after the other; two blocks per SM
constexpr int PREP_FLOATS = 2 * GC * GD + 2 * GC * GC + 32 * 32;
constexpr int PREP_GROUP_MAX = 8;      // value heads per key head whose decays fit the block's tables

__global__ void __launch_bounds__(256, 2) gdn_chunk_prep_kernel(const GdnChunkParams p) {
    extern __shared__ float4 gsm4[];
    float *sK = reinterpret_cast<float *>(gsm4), *sQ = sK + GC * GD;          // V takes Q's place once the q . k products are in registers
    float *sA = sQ + GC * GD, *sT = sA + GC * GC, *sX = sT + GC * GC;
    __shared__ __align__(16) float sG[PREP_GROUP_MAX][GC], sR[PREP_GROUP_MAX][GC], sB[PREP_GROUP_MAX][GC], sE[GC];
    const int c = blockIdx.x, kh = blockIdx.y, b = blockIdx.z, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int key_dim = (p.nh / p.kv_group) * GD, val_dim = p.nh * GD, qkv_dim = 2 * key_dim + val_dim;
    const int64_t pos0 = (int64_t)b * p.n + (int64_t)c * GC;
    const int valid = min(GC, p.left - c * GC);
    const float *row0 = p.up + pos0 * qkv_dim;
    for (int x = tid; x < GC * (GD / 4); x += 256) {
        const int t = x >> 5, q = x & 31;
        const float *row = t < valid ? row0 + (int64_t)t * qkv_dim : row0;
        cp16(sK + piece<GD>(t, q), row + key_dim + (int64_t)kh * GD + q * 4, t < valid);
        cp16(sQ + piece<GD>(t, q), row + (int64_t)kh * GD + q * 4, t < valid);
    }
    cp_async_commit();
    for (int x = tid; x < p.kv_group * GC; x += 256) {
        const int g = x >> 6, t = x & 63, vh = kh * p.kv_group + g;
        float ld = 0.f, bt = 0.f;                            // a position past the end: no decay, nothing written
        if (t < valid) {
            const float ea = gc_exp(p.a_log[vh]);
            const float v = p.gdec[(pos0 + t) * p.nh + vh] + p.dt_bias[vh];
            const float sp = v > 20.0f ? v : (float)log1p((double)gc_exp(v));
            ld = -ea * sp;                                   // log of the position's decay
            bt = 1.0f / (1.0f + gc_exp(-p.beta[(pos0 + t) * p.nh + vh]));
        }
        sG[g][t] = ld;
        sB[g][t] = bt;
    }
    __syncthreads();
    // Running sums inside the chunk, two positions per lane. What is wanted is their differences, which are small where the
    // sums are large: sums in double, kept as a float and its remainder.
    for (int g = warp; g < p.kv_group; g += 8) {
        const double l0 = sG[g][2 * lane], l1 = sG[g][2 * lane + 1];
        double s = l0 + l1;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double u = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += u;
        }
        const double g0 = s - l1;
        const float h0 = (float)g0, h1 = (float)s;
        sG[g][2 * lane] = h0; sG[g][2 * lane + 1] = h1;
        sR[g][2 * lane] = (float)(g0 - h0); sR[g][2 * lane + 1] = (float)(s - h1);
    }
    cp_async_wait<0>();
    __syncthreads();
    // k_t . k_s and q_t . k_s in 16 x 16 blocks on and below the diagonal: a warp has row block rb and column blocks `half`
    // and half + 2, kept in registers; the two warps of a scheduler (w and w + 4) get three blocks or two between them.
    const int rb = warp < 4 ? warp : 7 - warp, half = warp >> 2, lg = lane >> 2, lt = lane & 3;
    float kk[2][2][4], qk[2][2][4];
#pragma unroll
    for (int u = 0; u < 2; u++) {
        const int sb = half + 2 * u;
#pragma unroll
        for (int n = 0; n < 2; n++)
#pragma unroll
            for (int i = 0; i < 4; i++) kk[u][n][i] = qk[u][n][i] = 0.f;
        if (sb > rb) continue;
        const RowPtrA pk = row_ptr_a<GD>(sK, rb * 16 + lg, lt), pq = row_ptr_a<GD>(sQ, rb * 16 + lg, lt);
        const RowPtr ps[2] = {row_ptr<GD>(sK, sb * 16 + lg, lt), row_ptr<GD>(sK, sb * 16 + 8 + lg, lt)};
#pragma unroll 2
        for (int k2 = 0; k2 < GD / 32; k2++) {
            Acc ak[2], aq[2];
            ak[0].zero(); ak[1].zero(); aq[0].zero(); aq[1].zero();
#pragma unroll
            for (int v = 0; v < 2; v++) {
                const OpA a = op_a(pk, 2 * k2 + v), q = op_a(pq, 2 * k2 + v);
#pragma unroll
                for (int n = 0; n < 2; n++) {
                    const OpB s = op_b(ps[n], 2 * k2 + v);
                    mma3(ak[n], a, s);
                    mma3(aq[n], q, s);
                }
            }
#pragma unroll
            for (int n = 0; n < 2; n++)
#pragma unroll
                for (int i = 0; i < 4; i++) { kk[u][n][i] += ak[n].sum(i); qk[u][n][i] += aq[n].sum(i); }
        }
    }

    for (int g = 0; g < p.kv_group; g++) {
        const int vh = kh * p.kv_group + g;
        float *w = ws_of(p, b, vh, c);
        __syncthreads();                                     // q's rows, or the head before's V and T, have been read
        for (int x = tid; x < GC * (GD / 4); x += 256) {
            const int t = x >> 5, q = x & 31;
            cp16(sQ + piece<GD>(t, q), (t < valid ? row0 + (int64_t)t * qkv_dim : row0) + 2 * key_dim + (int64_t)vh * GD + q * 4, t < valid);
        }
        cp_async_commit();
        if (tid < GC) {
            w[WS_G + tid] = sG[g][tid];
            w[WS_G + GC + tid] = sR[g][tid];
            sE[tid] = sB[g][tid] * expf(sG[g][tid]);
        }
        // A (strictly lower) and M (lower, with the diagonal; zeros above it)
#pragma unroll
        for (int u = 0; u < 2; u++)
#pragma unroll
            for (int n = 0; n < 2; n++)
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int t = rb * 16 + lg + 8 * h, s = (half + 2 * u) * 16 + n * 8 + 2 * lt;
                    const float gt = sG[g][t], rt = sR[g][t], bt = sB[g][t];
                    float a[2], m[2];
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        const float r = s + e <= t ? expf((gt - sG[g][s + e]) + (rt - sR[g][s + e])) : 0.f;
                        a[e] = s + e < t ? bt * r * kk[u][n][2 * h + e] : 0.f;
                        m[e] = r * qk[u][n][2 * h + e];
                    }
                    *reinterpret_cast<float2 *>(sA + piece<GC>(t, s >> 2) + (s & 3)) = make_float2(a[0], a[1]);
                    *reinterpret_cast<float2 *>(w + WS_M + t * GC + s) = make_float2(m[0], m[1]);
                }
        __syncthreads();
        // T = (I + A)^-1: the 16 x 16 blocks on the diagonal by forward substitution, a thread per column (the others clear the
        // two blocks above the diagonal that the last step reads); then the blocks below them, [X 0; B Y]^-1 = [X' 0; -Y' B X' Y'],
        // first at 16, then at 32, four columns per thread.
        if (tid < GC) {
            const int r = tid >> 4, col = tid & 15;
            float v[16];
#pragma unroll
            for (int t = 0; t < 16; t++) {
                float x = t == col ? 1.f : 0.f, y = 0.f;
#pragma unroll
                for (int s = 0; s < t; s++) {
                    const float a = sA[piece<GC>(16 * r + t, 4 * r + (s >> 2)) + (s & 3)];
                    if (s & 1) y -= a * v[s];
                    else x -= a * v[s];
                }
                v[t] = x + y;
            }
#pragma unroll
            for (int t = 0; t < 16; t++) sT[piece<GC>(16 * r + t, 4 * r + (col >> 2)) + (col & 3)] = v[t];
        } else if (tid < 192) {
            const int x = tid - 64, r = (x >> 6) * 32 + ((x >> 2) & 15);
            *reinterpret_cast<float4 *>(sT + piece<GC>(r, (r >> 5) * 8 + 4 + (x & 3))) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        __syncthreads();
        // row `row` of a [.. x 4 nq] block of P (pieces q0 ..) times a block whose rows are given by `get`
        auto quad = [&](const float *P, int row, int q0, int nq, auto get) -> float4 {
            float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
            for (int q = 0; q < nq; q++) {
                const float4 a = *reinterpret_cast<const float4 *>(P + piece<GC>(row, q0 + q));
                const float av[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const float4 x = get(4 * q + e);
                    o.x += av[e] * x.x; o.y += av[e] * x.y; o.z += av[e] * x.z; o.w += av[e] * x.w;
                }
            }
            return o;
        };
        auto neg = [](float4 v) { return make_float4(-v.x, -v.y, -v.z, -v.w); };
        {
            const int pr = tid >> 6, t = (tid >> 2) & 15, cq = tid & 3, r0 = 32 * pr;         // blocks (1, 0) and (3, 2): threads 0 .. 127
            if (tid < 128)
                *reinterpret_cast<float4 *>(sX + pr * 256 + t * 16 + cq * 4) =
                    quad(sA, r0 + 16 + t, r0 / 4, 4, [&](int s) { return *reinterpret_cast<const float4 *>(sT + piece<GC>(r0 + s, r0 / 4 + cq)); });
            __syncthreads();
            if (tid < 128)
                *reinterpret_cast<float4 *>(sT + piece<GC>(r0 + 16 + t, r0 / 4 + cq)) =
                    neg(quad(sT, r0 + 16 + t, r0 / 4 + 4, 4, [&](int s) { return *reinterpret_cast<const float4 *>(sX + pr * 256 + s * 16 + cq * 4); }));
            __syncthreads();
        }
        {
            const int t = tid >> 3, cq = tid & 7;                                             // the lower left 32 x 32: every thread
            *reinterpret_cast<float4 *>(sX + t * 32 + cq * 4) =
                quad(sA, 32 + t, 0, 8, [&](int s) { return *reinterpret_cast<const float4 *>(sT + piece<GC>(s, cq)); });
            __syncthreads();
            *reinterpret_cast<float4 *>(sT + piece<GC>(32 + t, cq)) =
                neg(quad(sT, 32 + t, 8, 8, [&](int s) { return *reinterpret_cast<const float4 *>(sX + s * 32 + cq * 4); }));
            __syncthreads();
        }
        // T diag(beta e^G) in A's place, T diag(beta) in T's
        for (int x = tid; x < GC * (GC / 4); x += 256) {
            const int t = x >> 4, q = x & 15, at = piece<GC>(t, q);
            const float4 v = *reinterpret_cast<const float4 *>(sT + at);
            const float4 bt = *reinterpret_cast<const float4 *>(&sB[g][4 * q]), be = *reinterpret_cast<const float4 *>(&sE[4 * q]);
            *reinterpret_cast<float4 *>(sA + at) = make_float4(v.x * be.x, v.y * be.y, v.z * be.z, v.w * be.w);
            *reinterpret_cast<float4 *>(sT + at) = make_float4(v.x * bt.x, v.y * bt.y, v.z * bt.z, v.w * bt.w);
        }
        cp_async_wait<0>();                                  // V
        __syncthreads();
        // W = T diag(beta e^G) K, and U~^T = V^T (T diag(beta))^T: 16 positions x 64 columns a warp; a row block's sums end
        // at its own diagonal (the two warps of a scheduler have complementary row blocks).
        {
            Acc acc[8];
#pragma unroll
            for (int n = 0; n < 8; n++) acc[n].zero();
            const RowPtrA pa = row_ptr_a<GC>(sA, rb * 16 + lg, lt);
#pragma unroll 1
            for (int k = 0; k <= rb; k++) {
                const OpA a = op_a(pa, k);
#pragma unroll
                for (int n = 0; n < 8; n++) {
                    float v[4];
                    col4<GD>(v, col_ptr<GD>(sK + k * 16 * GD, half * 64 + n * 8 + lg, lt), 0);
                    mma3(acc[n], a, op_b(v));
                }
            }
#pragma unroll
            for (int n = 0; n < 8; n++)
#pragma unroll
                for (int h = 0; h < 2; h++)
                    *reinterpret_cast<float2 *>(w + (rb * 16 + lg + 8 * h) * GD + half * 64 + n * 8 + 2 * lt) = make_float2(acc[n].sum(2 * h), acc[n].sum(2 * h + 1));
        }
        {
            Acc acc[4][2];
#pragma unroll
            for (int m = 0; m < 4; m++) { acc[m][0].zero(); acc[m][1].zero(); }
            const RowPtr pb0 = row_ptr<GC>(sT, rb * 16 + lg, lt), pb1 = row_ptr<GC>(sT, rb * 16 + 8 + lg, lt);
#pragma unroll 1
            for (int k = 0; k <= rb; k++) {
                const OpB b0 = op_b(pb0, k), b1 = op_b(pb1, k);
#pragma unroll
                for (int m = 0; m < 4; m++) {
                    float r0[4], r1[4];
                    col4<GD>(r0, col_ptr<GD>(sQ + k * 16 * GD, half * 64 + m * 16 + lg, lt), 0);
                    col4<GD>(r1, col_ptr<GD>(sQ + k * 16 * GD, half * 64 + m * 16 + 8 + lg, lt), 0);
                    const OpA a = op_a(r0, r1);
                    mma3(acc[m][0], a, b0);
                    mma3(acc[m][1], a, b1);
                }
            }
#pragma unroll
            for (int m = 0; m < 4; m++)
#pragma unroll
                for (int n = 0; n < 2; n++)
#pragma unroll
                    for (int h = 0; h < 2; h++)
                        *reinterpret_cast<float2 *>(w + WS_U + (half * 64 + m * 16 + lg + 8 * h) * GC + rb * 16 + n * 8 + 2 * lt) =
                            make_float2(acc[m][n].sum(2 * h), acc[m][n].sum(2 * h + 1));
        }
    }
}

// ---- scan: grid (32-column block of the value dimension, value head, slot), 256 threads; chunks in order. Everything is
// transposed, rows = value columns: U^T = U~^T - S0 W^T and S0 <- e^(G_64) S0 + (U^T diag(e^(G_64 - G))) K. A thread keeps
// its piece of the state in registers from the first chunk to the last; shared memory has the copy that the first product
// reads. W and K of the next chunk arrive by asynchronous copies under this chunk's arithmetic, U~ and G in registers.
constexpr int SCAN_FLOATS = 4 * GC * GD + GD * GJ + GC * GJ;

__global__ void __launch_bounds__(256, 1) gdn_chunk_scan_kernel(const GdnChunkParams p) {
    extern __shared__ float4 gsm4[];
    float *sW = reinterpret_cast<float *>(gsm4), *sK = sW + 2 * GC * GD;      // two [64][128] tiles each
    float *sS = sK + 2 * GC * GD, *sU = sS + GD * GJ;                         // S0 [32 value][128 key]; (e^(G_64 - G) U)^T [32 value][64]
    const int jb = blockIdx.x, vh = blockIdx.y, b = blockIdx.z, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int lg = lane >> 2, lt = lane & 3;
    const int kh = vh / p.kv_group;
    const int key_dim = (p.nh / p.kv_group) * GD, val_dim = p.nh * GD, qkv_dim = 2 * key_dim + val_dim;
    // this thread's sixteen bytes of rows warp, warp + 8, ..: their places alternate between two permutations
    const int at0 = piece<GD>(warp, lane), at1 = piece<GD>(warp + 8, lane) - 8 * GD;
    const float *wsrc = ws_of(p, b, vh, 0) + warp * GD + lane * 4;
    const float *ksrc = p.up + ((int64_t)b * p.n + warp) * qkv_dim + key_dim + (int64_t)kh * GD + lane * 4;
    auto issue = [&](int c) {                              // chunks in order
        if (c < p.nchunks) {
            const int valid = p.left - c * GC - warp;
            float *dw = sW + (c & 1) * GC * GD, *dk = sK + (c & 1) * GC * GD;
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const int at = ((i & 1) ? at1 : at0) + i * 8 * GD;
                cp16(dw + at, wsrc + i * 8 * GD, true);
                cp16(dk + at, 8 * i < valid ? ksrc + (int64_t)(8 * i) * qkv_dim : wsrc, 8 * i < valid);      // (past the end: any address that can be read)
            }
            ksrc += (int64_t)GC * qkv_dim;
            wsrc += WS_PER;
        }
        cp_async_commit();
    };
    issue(0);
    const int v0 = (warp & 1) * 16, p0 = (warp >> 1) * 16;                                // first product: values v0 .. + 15, positions p0 .. + 15
    const int k0 = warp * 16;                                                             // second product: all 32 values, keys k0 .. + 15
    float *Sh = p.S + (((int64_t)b * p.nh + vh) * GD + (int64_t)jb * GJ) * GD;           // rows jb*32 .. +31 of the head's [value][key] state
    float S[2][2][4];                                                                     // [16-value block][8-key block]: value lg (+ 8), keys 2 lt, 2 lt + 1
    auto put_state = [&]() {
#pragma unroll
        for (int m = 0; m < 2; m++)
#pragma unroll
            for (int n = 0; n < 2; n++)
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int v = m * 16 + lg + 8 * h, k = k0 + n * 8 + 2 * lt;
                    *reinterpret_cast<float2 *>(sS + piece<GD>(v, k >> 2) + (k & 3)) = make_float2(S[m][n][2 * h], S[m][n][2 * h + 1]);
                }
    };
#pragma unroll
    for (int m = 0; m < 2; m++)
#pragma unroll
        for (int n = 0; n < 2; n++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const float2 f = *reinterpret_cast<const float2 *>(Sh + (int64_t)(m * 16 + lg + 8 * h) * GD + k0 + n * 8 + 2 * lt);
                S[m][n][2 * h] = f.x; S[m][n][2 * h + 1] = f.y;
            }
    put_state();
    float2 u[2][2], gp[2], gr[2];                          // U~ of this lane: [8-position block][value lg, lg + 8]; G there and its remainder
    float gl, glr;
    auto fetch = [&](int c) {
        const float *w = ws_of(p, b, vh, c);
#pragma unroll
        for (int n = 0; n < 2; n++) {
#pragma unroll
            for (int h = 0; h < 2; h++) u[n][h] = *reinterpret_cast<const float2 *>(w + WS_U + (jb * GJ + v0 + lg + 8 * h) * GC + p0 + n * 8 + 2 * lt);
            gp[n] = *reinterpret_cast<const float2 *>(w + WS_G + p0 + n * 8 + 2 * lt);
            gr[n] = *reinterpret_cast<const float2 *>(w + WS_G + GC + p0 + n * 8 + 2 * lt);
        }
        gl = w[WS_G + GC - 1];
        glr = w[WS_G + 2 * GC - 1];
    };
    fetch(0);
    const RowPtrA pS = row_ptr_a<GD>(sS, v0 + lg, lt), pU0 = row_ptr_a<GC>(sU, lg, lt), pU1 = row_ptr_a<GC>(sU, 16 + lg, lt);
    const RowPtr pW[2] = {row_ptr<GD>(sW, p0 + lg, lt), row_ptr<GD>(sW, p0 + 8 + lg, lt)};
    const ColPtr pK[2] = {col_ptr<GD>(sK, k0 + lg, lt), col_ptr<GD>(sK, k0 + 8 + lg, lt)};
    for (int c = 0; c < p.nchunks; c++) {
        float *w = ws_of(p, b, vh, c);
        const int odd = (c & 1) * GC * GD;
        cp_async_wait<0>();
        __syncthreads();                                   // W and K of this chunk and the state are in place; the other tiles are free
        issue(c + 1);
        // the state at the chunk's start, for the output kernel
        for (int x = tid; x < GJ * (GD / 4); x += 256) {
            const int j = x >> 5, q = x & 31;
            *reinterpret_cast<float4 *>(w + WS_S + (jb * GJ + j) * GD + q * 4) = *reinterpret_cast<const float4 *>(sS + piece<GD>(j, q));
        }
        float d[2][4];
#pragma unroll
        for (int n = 0; n < 2; n++)
#pragma unroll
            for (int i = 0; i < 4; i++) d[n][i] = 0.f;
#pragma unroll
        for (int k2 = 0; k2 < GD / 32; k2++) {
            Acc acc[2];
            acc[0].zero(); acc[1].zero();
#pragma unroll
            for (int v = 0; v < 2; v++) {
                const OpA a = op_a(pS, 2 * k2 + v);
#pragma unroll
                for (int n = 0; n < 2; n++) mma3(acc[n], a, op_b(RowPtr{{pW[n].p[0] + odd, pW[n].p[1] + odd}}, 2 * k2 + v));
            }
#pragma unroll
            for (int n = 0; n < 2; n++)
#pragma unroll
                for (int i = 0; i < 4; i++) d[n][i] += acc[n].sum(i);
        }
        const float dl = expf(gl);
#pragma unroll
        for (int n = 0; n < 2; n++) {
            const float f0 = expf((gl - gp[n].x) + (glr - gr[n].x)), f1 = expf((gl - gp[n].y) + (glr - gr[n].y));
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int v = v0 + lg + 8 * h, t = p0 + n * 8 + 2 * lt;
                const float2 x = make_float2(u[n][h].x - d[n][2 * h], u[n][h].y - d[n][2 * h + 1]);
                *reinterpret_cast<float2 *>(w + WS_U + (jb * GJ + v) * GC + t) = x;
                *reinterpret_cast<float2 *>(sU + piece<GC>(v, t >> 2) + (t & 3)) = make_float2(x.x * f0, x.y * f1);
            }
        }
        if (c + 1 < p.nchunks) fetch(c + 1);
        __syncthreads();                                   // U is in place; the state has been read
#pragma unroll
        for (int m = 0; m < 2; m++)
#pragma unroll
            for (int n = 0; n < 2; n++)
#pragma unroll
                for (int i = 0; i < 4; i++) S[m][n][i] *= dl;
#pragma unroll
        for (int k2 = 0; k2 < GC / 32; k2++) {
            Acc acc[2][2];
#pragma unroll
            for (int m = 0; m < 2; m++) { acc[m][0].zero(); acc[m][1].zero(); }
#pragma unroll
            for (int v = 0; v < 2; v++) {
                const OpA a0 = op_a(pU0, 2 * k2 + v), a1 = op_a(pU1, 2 * k2 + v);
#pragma unroll
                for (int n = 0; n < 2; n++) {
                    float x[4];
#pragma unroll
                    for (int e = 0; e < 4; e++) x[e] = pK[n].p[e][odd + (2 * k2 + v) * 16 * GD];
                    const OpB kb = op_b(x);
                    mma3(acc[0][n], a0, kb);
                    mma3(acc[1][n], a1, kb);
                }
            }
#pragma unroll
            for (int m = 0; m < 2; m++)
#pragma unroll
                for (int n = 0; n < 2; n++)
#pragma unroll
                    for (int i = 0; i < 4; i++) S[m][n][i] += acc[m][n].sum(i);
        }
        put_state();
    }
#pragma unroll
    for (int m = 0; m < 2; m++)
#pragma unroll
        for (int n = 0; n < 2; n++)
#pragma unroll
            for (int h = 0; h < 2; h++)
                *reinterpret_cast<float2 *>(Sh + (int64_t)(m * 16 + lg + 8 * h) * GD + k0 + n * 8 + 2 * lt) = make_float2(S[m][n][2 * h], S[m][n][2 * h + 1]);
}

// ---- output: persistent blocks of 512 threads take (chunk, head) items in turn. O = diag(e^G) Q S0^T + M U for all 64
// positions x 128 value columns at once, then the gated RMS norm of every row (:1250-1262). The operands stream through a
// ring of six 24 KB stages of 32 contraction terms -- four of Q and S0, two of M and U, the next item's behind them -- so that
// memory works under the arithmetic and across items.
constexpr int OUT_STAGES = 6, OUT_STAGE_FLOATS = (GC + GD) * 32;          // as many stages as steps: step i of every item uses stage i

__global__ void __launch_bounds__(512, 1) gdn_chunk_out_kernel(const GdnChunkParams p, int items) {
    extern __shared__ float4 gsm4[];
    float *ring = reinterpret_cast<float *>(gsm4);           // stage: A [64 position][32] | B [128 value][32]
    __shared__ float sR[8][GC];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, lg = lane >> 2, lt = lane & 3;
    const int key_dim = (p.nh / p.kv_group) * GD, val_dim = p.nh * GD, qkv_dim = 2 * key_dim + val_dim;
    const int t0 = (warp & 1) * 32, j0 = (warp >> 1) * 16;   // a warp has 32 positions x 16 columns
    // the copies: this thread's sixteen bytes of rows cr (positions) and cr, cr + 64 (value columns) of a stage
    const int cr = tid >> 3, cq = (tid & 7) * 4, at = piece<32>(cr, tid & 7);
    int li = blockIdx.x;                                     // the item being loaded, and where its operands are
    const float *lw = nullptr, *lq = nullptr;
    bool lvalid = false;
    auto open_item = [&]() {
        if (li >= items) return;
        const int c = li % p.nchunks, bh = li / p.nchunks, vh = bh % p.nh, b = bh / p.nh;      // (slot, head, chunk) with the chunk fastest
        lw = p.ws + (int64_t)li * WS_PER;
        lvalid = cr < p.left - c * GC;
        lq = p.up + ((int64_t)b * p.n + (int64_t)c * GC + (lvalid ? cr : 0)) * qkv_dim + (int64_t)(vh / p.kv_group) * GD + cq;
    };
    auto issue = [&](int step) {
        if (li < items) {
            float *dst = ring + step * OUT_STAGE_FLOATS + at;
            if (step < 4) {
                cp16(dst, lq + step * 32, lvalid);
                cp16(dst + GC * 32, lw + WS_S + cr * GD + cq + step * 32, true);
                cp16(dst + 2 * GC * 32, lw + WS_S + (cr + 64) * GD + cq + step * 32, true);
            } else {
                cp16(dst, lw + WS_M + cr * GC + cq + (step - 4) * 32, true);
                cp16(dst + GC * 32, lw + WS_U + cr * GC + cq + (step - 4) * 32, true);
                cp16(dst + 2 * GC * 32, lw + WS_U + (cr + 64) * GC + cq + (step - 4) * 32, true);
            }
        }
        cp_async_commit();
    };
    open_item();
#pragma unroll
    for (int n = 0; n < OUT_STAGES - 1; n++) issue(n);
    const RowPtrA pA[2] = {row_ptr_a<32>(ring, t0 + lg, lt), row_ptr_a<32>(ring, t0 + 16 + lg, lt)};
    const RowPtr pB[2] = {row_ptr<32>(ring + GC * 32, j0 + lg, lt), row_ptr<32>(ring + GC * 32, j0 + 8 + lg, lt)};
    for (int item = blockIdx.x; item < items; item += gridDim.x) {
        const int c = item % p.nchunks, bh = item / p.nchunks, vh = bh % p.nh, b = bh / p.nh;
        const float *w = p.ws + (int64_t)item * WS_PER;
        float r[2][2][4], eg[2][2];
#pragma unroll
        for (int m = 0; m < 2; m++) {
#pragma unroll
            for (int h = 0; h < 2; h++) eg[m][h] = w[WS_G + t0 + m * 16 + lg + 8 * h];
#pragma unroll
            for (int k = 0; k < 2; k++)
#pragma unroll
                for (int i = 0; i < 4; i++) r[m][k][i] = 0.f;
        }
#pragma unroll
        for (int step = 0; step < OUT_STAGES; step++) {
            cp_async_wait<OUT_STAGES - 2>();
            __syncthreads();                                 // this step's operands are here; every warp is done with the step before
            if (step == 1) { li += gridDim.x; open_item(); } // (the step before this one was the last of the item to be asked for)
            issue(step == 0 ? OUT_STAGES - 1 : step - 1);
            if (step == 4) {
#pragma unroll
                for (int m = 0; m < 2; m++)
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const float e = expf(eg[m][h]);
#pragma unroll
                        for (int k = 0; k < 2; k++) { r[m][k][2 * h] *= e; r[m][k][2 * h + 1] *= e; }
                    }
            }
            if (step == 5 && t0 == 0) continue;              // (positions 32 .. 63 are in no sum of the first 32 rows)
            Acc acc[2][2];
#pragma unroll
            for (int m = 0; m < 2; m++) { acc[m][0].zero(); acc[m][1].zero(); }
#pragma unroll
            for (int v = 0; v < 2; v++) {
                auto shift = [&](const RowPtr &x) { return RowPtr{{x.p[0] + step * OUT_STAGE_FLOATS, x.p[1] + step * OUT_STAGE_FLOATS}}; };
                const OpB b0 = op_b(shift(pB[0]), v), b1 = op_b(shift(pB[1]), v);
#pragma unroll
                for (int m = 0; m < 2; m++) {
                    const OpA a = op_a(RowPtrA{shift(pA[m].r0), shift(pA[m].r1)}, v);
                    mma3(acc[m][0], a, b0);
                    mma3(acc[m][1], a, b1);
                }
            }
#pragma unroll
            for (int m = 0; m < 2; m++)
#pragma unroll
                for (int k = 0; k < 2; k++)
#pragma unroll
                    for (int i = 0; i < 4; i++) r[m][k][i] += acc[m][k].sum(i);
        }
        const int64_t pos0 = (int64_t)b * p.n + (int64_t)c * GC;
        const int valid = min(GC, p.left - c * GC);
#pragma unroll
        for (int m = 0; m < 2; m++)
#pragma unroll
            for (int h = 0; h < 2; h++) {                    // a row's squares: its four lanes, then the eight warps that share it
                float v = (r[m][0][2 * h] * r[m][0][2 * h] + r[m][0][2 * h + 1] * r[m][0][2 * h + 1]) +
                          (r[m][1][2 * h] * r[m][1][2 * h] + r[m][1][2 * h + 1] * r[m][1][2 * h + 1]);
                v += __shfl_xor_sync(0xffffffffu, v, 1);
                v += __shfl_xor_sync(0xffffffffu, v, 2);
                if (lt == 0) sR[warp >> 1][t0 + m * 16 + lg + 8 * h] = v;
            }
        float2 z[2][2][2], nw[2];
#pragma unroll
        for (int k = 0; k < 2; k++) {
            nw[k] = *reinterpret_cast<const float2 *>(p.norm + j0 + k * 8 + 2 * lt);
#pragma unroll
            for (int m = 0; m < 2; m++)
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int t = t0 + m * 16 + lg + 8 * h;
                    z[m][h][k] = t < valid ? *reinterpret_cast<const float2 *>(p.gate + (pos0 + t) * val_dim + (int64_t)vh * GD + j0 + k * 8 + 2 * lt) : make_float2(0.f, 0.f);
                }
        }
        __syncthreads();
#pragma unroll
        for (int m = 0; m < 2; m++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int t = t0 + m * 16 + lg + 8 * h;
                float ss = 0.f;
#pragma unroll
                for (int i = 0; i < 8; i++) ss += sR[i][t];
                if (t >= valid) continue;
                const float rstd = 1.0f / sqrtf(ss / (float)GD + p.rms_eps);
#pragma unroll
                for (int k = 0; k < 2; k++) {
                    const float2 zz = z[m][h][k];
                    *reinterpret_cast<float2 *>(p.out + (pos0 + t) * val_dim + (int64_t)vh * GD + j0 + k * 8 + 2 * lt) =
                        make_float2(r[m][k][2 * h] * (rstd * nw[k].x * (zz.x / (1.0f + expf(-zz.x)))), r[m][k][2 * h + 1] * (rstd * nw[k].y * (zz.y / (1.0f + expf(-zz.y)))));
                }
            }
    }
    cp_async_wait<0>();
}

}  // namespace

// Whether the chunk-parallel kernels take the call: their vector accesses want 16-byte aligned arrays.
bool cwk_gdn_chunked_ok(int kv_group, const float *up, const float *gate, const float *norm, const float *S, const float *out) {
    return kv_group <= PREP_GROUP_MAX && ((reinterpret_cast<uintptr_t>(up) | reinterpret_cast<uintptr_t>(gate) | reinterpret_cast<uintptr_t>(norm) |
                                           reinterpret_cast<uintptr_t>(S) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
}

int cwk_gdn_scan_chunked(cwk_ctx *ctx, int B, int n, int nh, int kv_group, const float *up, const float *gdec, const float *beta, const float *gate,
                         const float *a_log, const float *dt_bias, const float *norm, float rms_eps, float *S, float *out) {
    // Segments of chunks, one after another, and groups of slots where there are many: the workspace is bounded whatever the
    // prompt's length, and the state goes from segment to segment in S.
    const int all = (n + GC - 1) / GC;
    const auto even = [](int total, int64_t most) {        // as few parts of at most `most` as it takes, alike
        const int parts = (int)((total + most - 1) / most);
        return (total + parts - 1) / parts;
    };
    constexpr int64_t room = WS_MAX / (WS_PER * (int64_t)sizeof(float));
    const int nb = even(B, std::max<int64_t>(1, std::min<int64_t>(B, room / ((int64_t)nh * std::min(all, 8)))));
    const int seg = even(all, std::max<int64_t>(1, std::min<int64_t>(all, room / ((int64_t)nh * nb))));
    int s = cwk_reserve_work(ctx, (size_t)nb * nh * seg * WS_PER * sizeof(float));
    if (s != CWK_OK) return s;
    static bool attr_set[16] = {false};
    if (!attr_set[ctx->device & 15]) {
        CWK_CUDA(ctx, cudaFuncSetAttribute(gdn_chunk_prep_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, PREP_FLOATS * 4));
        CWK_CUDA(ctx, cudaFuncSetAttribute(gdn_chunk_scan_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SCAN_FLOATS * 4));
        CWK_CUDA(ctx, cudaFuncSetAttribute(gdn_chunk_out_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, OUT_STAGES * OUT_STAGE_FLOATS * 4));
        attr_set[ctx->device & 15] = true;
    }
    const int64_t val_dim = (int64_t)nh * GD, qkv_dim = 2 * (int64_t)(nh / kv_group) * GD + val_dim;
    GdnChunkParams p;
    p.a_log = a_log; p.dt_bias = dt_bias; p.norm = norm; p.ws = (float *)ctx->work; p.n = n; p.nh = nh; p.kv_group = kv_group; p.rms_eps = rms_eps;
    for (int b0 = 0; b0 < B; b0 += nb) {
        const int slots = std::min(nb, B - b0);
        p.S = S + (int64_t)b0 * nh * GD * GD;
        for (int c0 = 0; c0 < all; c0 += seg) {
            const int64_t at = (int64_t)b0 * n + (int64_t)c0 * GC;
            p.up = up + at * qkv_dim; p.gdec = gdec + at * nh; p.beta = beta + at * nh; p.gate = gate + at * val_dim; p.out = out + at * val_dim;
            p.left = n - c0 * GC; p.nchunks = std::min(seg, all - c0);
            gdn_chunk_prep_kernel<<<dim3(p.nchunks, nh / kv_group, slots), 256, PREP_FLOATS * 4, ctx->stream>>>(p);
            CWK_LAUNCH_CHECK(ctx, "gdn_chunk_prep_kernel");
            {
                CwkKernelTimer timer(ctx);
                gdn_chunk_scan_kernel<<<dim3(GD / GJ, nh, slots), 256, SCAN_FLOATS * 4, ctx->stream>>>(p);
                CWK_LAUNCH_CHECK(ctx, "gdn_chunk_scan_kernel");
            }
            const int items = slots * nh * p.nchunks;
            gdn_chunk_out_kernel<<<std::min(items, ctx->sm_count), 512, OUT_STAGES * OUT_STAGE_FLOATS * 4, ctx->stream>>>(p, items);
            CWK_LAUNCH_CHECK(ctx, "gdn_chunk_out_kernel");
        }
    }
    return CWK_OK;
}
