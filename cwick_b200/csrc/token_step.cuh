// token_step.cuh -- kernels of the reference-named decode call for one token (src/attention.c:642-902), included by dropin.cu
// behind its projection helpers.
//
// A token's projections are their weights read once: 126 MB in BF16 for a layer of hidden 4096, 19 us of HBM time. What a
// chain of eight kernels adds to that is latency -- a kernel comes up, asks for its first bytes, waits a microsecond, and at
// its end HBM idles until the next one has done the same (100 us per call). So here every kernel (1) comes up while the one
// before still runs (cwk_launch_early) and asks for its first weights, which depend on nothing, before it waits for its
// activations; and (2) small steps ride along: the two norms in the q_b projection's blocks, the merge of the attention's
// split records in the un-absorb. (Telling L2 from the first projection and from the attention to fetch the weights that
// come next made a call 1 to 3 us longer.)
#pragma once

// y[r] = W[r] . x for one token (as gemv_rows_kernel, rows of whole 16-byte pieces only). The grid is what fits on the SMs at
// once, two blocks of sixteen warps each, and a block goes through a contiguous range of rows: with a block per few rows, a
// second wave of blocks came up in the middle of every projection, each asking for its first bytes anew (q_b 12 us, now 6).
// wpr warps share a pair of rows, so that an activation read from shared memory or L1 meets two weights (at one, those
// reads take as long as HBM needs for the weights), chosen so that the rounds come out even. A block's results leave together: the
// last projection's go to host memory, and a row of its own is a bus transaction of four bytes.
// What x is: X_PLAIN as it is; X_NORM x / sqrt(mean(x^2) + eps) * w, worked out by every block for itself; X_SUM x + x2. In the
// last two the values are kept in shared memory. X_NORM: the launch's last block is not a projection block but does the
// kv_a row: normalised in place, narrowed into the cache row and written to the caller's staging.
enum { X_PLAIN = 0, X_NORM = 1, X_SUM = 2 };
struct TokenInput {
    const float *x, *x2;
    const uint16_t *w, *wkv;
    float eps;
    float *kva;
    int nkv;
    uint16_t *row_out;
    void *host_row;
    int host_bf16;
};
constexpr int TG_WARPS = 16, TG_MAX_ROWS = 512;      // rows per block (a block's results wait in shared memory)
template <int KIND, int XIN>
__global__ void __launch_bounds__(32 * TG_WARPS, 2) gemv_token_kernel(const void *Wv, const float *scales, float *y, int rows, int k, int wpr, int blocks,
                                                                     const void *W2, const float *scales2, float *y2, int rows2, const TokenInput in) {
    constexpr int E = KIND == GEMV_BF16 ? 8 : KIND == GEMV_F32 ? 4 : 16, EB = 16 / E, AHEAD = 4;
    extern __shared__ __align__(16) float s_x[];
    __shared__ float s_part[2][TG_WARPS][2], s_y[TG_MAX_ROWS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    cwk_pdl_launch();
    if (XIN == X_NORM && blockIdx.x == blocks) {
        cwk_pdl_wait();
        if (threadIdx.x < 256) rms_scale_row(in.kva, in.nkv, in.wkv, in.eps, in.row_out, in.host_row, in.host_bf16);
        return;
    }
    const int slots = TG_WARPS / wpr, slot = warp / wpr, part = warp % wpr;      // pairs at a time; this warp's pair and share of it
    const int step = wpr * 32 * E, j0 = (part * 32 + lane) * E;
    const int all = rows + rows2, lo = (int)((int64_t)all * blockIdx.x / blocks), hi = (int)((int64_t)all * (blockIdx.x + 1) / blocks);
    uint4 v[2][AHEAD];
    const uint8_t *w[2] = {nullptr, nullptr};
    const float *sc[2] = {nullptr, nullptr};
    int r = lo + 2 * slot;
    auto ask = [&]() {                                     // the first pieces of rows r and r + 1 (an odd last one twice)
        if (r >= hi) return;
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const int q = min(r + i, hi - 1);
            const bool second = q >= rows;
            const int rr = second ? q - rows : q;
            w[i] = reinterpret_cast<const uint8_t *>(second ? W2 : Wv) + (int64_t)rr * k * EB;
            if (KIND == GEMV_FP8) sc[i] = (second ? scales2 : scales) + (int64_t)(rr / 128) * ((k + 127) / 128);
#pragma unroll
            for (int u = 0; u < AHEAD; u++)
                if (j0 + u * step < k) v[i][u] = ld_weight16(w[i] + (int64_t)(j0 + u * step) * EB);
        }
    };
    ask();
    constexpr int NW = 4;                                  // activations at a time, and norm weights asked for ahead
    uint16_t nw[NW];
    if (XIN == X_NORM) {
#pragma unroll
        for (int u = 0; u < NW; u++) nw[u] = threadIdx.x + u * 32 * TG_WARPS < k ? in.w[threadIdx.x + u * 32 * TG_WARPS] : (uint16_t)0;
    }
    cwk_pdl_wait();
    const float *x = in.x;
    if (XIN == X_NORM) {
        __shared__ double s_ss[TG_WARPS];
        double ss = 0.0;
        for (int i = threadIdx.x; i < k; i += NW * 32 * TG_WARPS) {
            float f[NW];
#pragma unroll
            for (int u = 0; u < NW; u++) f[u] = i + u * 32 * TG_WARPS < k ? x[i + u * 32 * TG_WARPS] : 0.f;
#pragma unroll
            for (int u = 0; u < NW; u++)
                if (i + u * 32 * TG_WARPS < k) {
                    s_x[i + u * 32 * TG_WARPS] = f[u];     // (each thread scales what it wrote)
                    ss += (double)f[u] * (double)f[u];
                }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        if (lane == 0) s_ss[warp] = ss;
        __syncthreads();
        double tot = s_ss[lane & (TG_WARPS - 1)];
#pragma unroll
        for (int o = TG_WARPS / 2; o > 0; o >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, o);
        const float inv = __fdiv_rn(1.0f, (float)sqrt(tot / (double)k + (double)in.eps));
#pragma unroll
        for (int u = 0; u < NW; u++) {
            const int i = threadIdx.x + u * 32 * TG_WARPS;
            if (i < k) s_x[i] = s_x[i] * inv * bf16_bits_to_f32(nw[u]);
        }
        for (int i = threadIdx.x + NW * 32 * TG_WARPS; i < k; i += 32 * TG_WARPS) s_x[i] = s_x[i] * inv * bf16_bits_to_f32(in.w[i]);
        __syncthreads();
        x = s_x;
    } else if (XIN == X_SUM) {
        for (int i = threadIdx.x * 4; i < k; i += 2 * 128 * TG_WARPS) {      // two pieces of both at a time
            const bool two = i + 128 * TG_WARPS < k;
            float4 a[2], b[2];
#pragma unroll
            for (int u = 0; u < 2; u++)
                if (u == 0 || two) {
                    a[u] = *reinterpret_cast<const float4 *>(x + i + u * 128 * TG_WARPS);
                    b[u] = *reinterpret_cast<const float4 *>(in.x2 + i + u * 128 * TG_WARPS);
                }
#pragma unroll
            for (int u = 0; u < 2; u++)
                if (u == 0 || two)
                    *reinterpret_cast<float4 *>(s_x + i + u * 128 * TG_WARPS) = make_float4(a[u].x + b[u].x, a[u].y + b[u].y, a[u].z + b[u].z, a[u].w + b[u].w);
        }
        __syncthreads();
        x = s_x;
    }
    for (int it = 0; lo + it * 2 * slots < hi; it++) {     // (every warp of a block goes round as often)
        float acc[2] = {0.f, 0.f};
        const int row = r;
        if (r < hi) {
#pragma unroll
            for (int u = 0; u < AHEAD; u++)
                if (j0 + u * step < k) {
                    acc[0] += gemv_piece<KIND>(v[0][u], x, j0 + u * step, sc[0]);
                    acc[1] += gemv_piece<KIND>(v[1][u], x, j0 + u * step, sc[1]);
                }
            for (int j = j0 + AHEAD * step; j < k; j += AHEAD * step) {
#pragma unroll
                for (int u = 0; u < AHEAD; u++)
                    if (j + u * step < k) {
                        v[0][u] = ld_weight16(w[0] + (int64_t)(j + u * step) * EB);
                        v[1][u] = ld_weight16(w[1] + (int64_t)(j + u * step) * EB);
                    }
#pragma unroll
                for (int u = 0; u < AHEAD; u++)
                    if (j + u * step < k) {
                        acc[0] += gemv_piece<KIND>(v[0][u], x, j + u * step, sc[0]);
                        acc[1] += gemv_piece<KIND>(v[1][u], x, j + u * step, sc[1]);
                    }
            }
        }
        r += 2 * slots;
        ask();                                             // the next pair's pieces, under this one's sums
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], o);
            acc[1] += __shfl_xor_sync(0xffffffffu, acc[1], o);
        }
        if (wpr > 1) {
            if (lane == 0) { s_part[it & 1][warp][0] = acc[0]; s_part[it & 1][warp][1] = acc[1]; }
            __syncthreads();
            acc[0] = acc[1] = 0.f;
            for (int i = 0; i < wpr; i++) { acc[0] += s_part[it & 1][slot * wpr + i][0]; acc[1] += s_part[it & 1][slot * wpr + i][1]; }
        }
        if (part == 0 && lane < 2 && row + lane < hi) s_y[row + lane - lo] = acc[lane];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < hi - lo; i += 32 * TG_WARPS) (lo + i < rows ? y[lo + i] : y2[lo + i - rows]) = s_y[i];
}
bool gemv_token_ok(const cwk_ctx *ctx, const WeightMirror *w) {
    const int E = w->kind == CWKC_WEIGHT_BF16 ? 8 : w->kind == CWKC_WEIGHT_F32 ? 4 : 16;
    return w->cols % E == 0 && (reinterpret_cast<uintptr_t>(w->data) & 15) == 0 && w->rows <= (int64_t)TG_MAX_ROWS * ctx->sm_count;
}
// w2 != NULL: a second matrix of the same kind and width, in the same launch (X_PLAIN).
cudaError_t gemv_token(cwk_ctx *ctx, const WeightMirror *w, float *y, const WeightMirror *w2, float *y2, int xin, const TokenInput &in) {
    const int64_t rows2 = w2 ? w2->rows : 0, all = w->rows + rows2;
    const int E = w->kind == CWKC_WEIGHT_BF16 ? 8 : w->kind == CWKC_WEIGHT_F32 ? 4 : 16;
    const int pieces = (int)(w->cols / E);                 // of a row
    const int cap = 2 * ctx->sm_count - (xin == X_NORM ? 1 : 0);      // blocks that are resident together
    const int blocks = (int)std::min<int64_t>((all + 1) / 2, cap);
    const int64_t pairs = ((all + blocks - 1) / blocks + 1) / 2;
    int wpr = 1;
    int64_t best = -1;
    for (int c = 1; c <= TG_WARPS; c <<= 1) {              // least time of a block: rounds x (pieces per lane + what a round costs besides)
        const int64_t rounds = (pairs + TG_WARPS / c - 1) / (TG_WARPS / c), cost = rounds * ((pieces + 32 * c - 1) / (32 * c) * 2 + (c > 1 ? 3 : 2));
        if (best < 0 || cost < best) { best = cost; wpr = c; }
    }
    auto go = [&](auto kern) {
        ctx->launches++;
        return cwk_launch_early(kern, dim3((unsigned)(blocks + (xin == X_NORM ? 1 : 0))), dim3(32 * TG_WARPS), xin == X_PLAIN ? 0 : (size_t)w->cols * 4, ctx->stream,
                                (const void *)w->data, (const float *)w->scales, y, (int)w->rows, (int)w->cols, wpr, blocks, (const void *)(w2 ? w2->data : nullptr),
                                (const float *)(w2 ? w2->scales : nullptr), y2, (int)rows2, in);
    };
    auto kinds = [&](auto bf16, auto f32, auto fp8) { return w->kind == CWKC_WEIGHT_BF16 ? go(bf16) : w->kind == CWKC_WEIGHT_F32 ? go(f32) : go(fp8); };
    if (xin == X_NORM) return kinds(gemv_token_kernel<GEMV_BF16, X_NORM>, gemv_token_kernel<GEMV_F32, X_NORM>, gemv_token_kernel<GEMV_FP8, X_NORM>);
    if (xin == X_SUM) return kinds(gemv_token_kernel<GEMV_BF16, X_SUM>, gemv_token_kernel<GEMV_F32, X_SUM>, gemv_token_kernel<GEMV_FP8, X_SUM>);
    return kinds(gemv_token_kernel<GEMV_BF16, X_PLAIN>, gemv_token_kernel<GEMV_F32, X_PLAIN>, gemv_token_kernel<GEMV_FP8, X_PLAIN>);
}

// q_abs[h][c] = sum_r q[h][r] W_k[h][r][c] (src/attention.c:741-744) for one token: grid (heads, kv_lora / 256), 512 threads,
// sixteen rows of 256 columns at a time, eight of them per thread on their way before q is there.
__global__ void __launch_bounds__(512) absorb_token_kernel(const float *q, const uint16_t *kvb, int nope, int kv_dim, int kv_lora, uint16_t *qabs) {
    __shared__ __align__(16) float s_sum[16][256];
    const int h = blockIdx.x, rg = threadIdx.x >> 5, c8 = (threadIdx.x & 31) * 8, col0 = blockIdx.y * 256;
    const uint16_t *wk = kvb + (int64_t)h * kv_dim * kv_lora + col0 + c8;
    cwk_pdl_launch();
    uint4 v[8];
#pragma unroll
    for (int u = 0; u < 8; u++)
        if (rg + 16 * u < nope) v[u] = ld_weight16(wk + (int64_t)(rg + 16 * u) * kv_lora);
    cwk_pdl_wait();
    q += (int64_t)h * nope;
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    auto fma8 = [&](const uint4 &x, float qv) {
        acc[0] += qv * __uint_as_float(x.x << 16); acc[1] += qv * __uint_as_float(x.x & 0xffff0000u);
        acc[2] += qv * __uint_as_float(x.y << 16); acc[3] += qv * __uint_as_float(x.y & 0xffff0000u);
        acc[4] += qv * __uint_as_float(x.z << 16); acc[5] += qv * __uint_as_float(x.z & 0xffff0000u);
        acc[6] += qv * __uint_as_float(x.w << 16); acc[7] += qv * __uint_as_float(x.w & 0xffff0000u);
    };
#pragma unroll
    for (int u = 0; u < 8; u++)
        if (rg + 16 * u < nope) fma8(v[u], q[rg + 16 * u]);
    for (int r = rg + 128; r < nope; r += 16) fma8(ld_weight16(wk + (int64_t)r * kv_lora), q[r]);
    *reinterpret_cast<float4 *>(&s_sum[rg][c8]) = make_float4(acc[0], acc[1], acc[2], acc[3]);
    *reinterpret_cast<float4 *>(&s_sum[rg][c8 + 4]) = make_float4(acc[4], acc[5], acc[6], acc[7]);
    __syncthreads();
    if (threadIdx.x < 256) {
        float t = 0.f;
#pragma unroll
        for (int g2 = 0; g2 < 16; g2++) t += s_sum[g2][threadIdx.x];
        qabs[(int64_t)h * kv_lora + col0 + threadIdx.x] = (uint16_t)(pack_bf16x2(t, 0.f) & 0xffffu);
    }
}

// The attention's split records of one token (nsplit <= 512 of [heads][512 + 2], flash_rows.cuh's layout) merged, and the
// result, rounded to bf16 as the merge on its own would leave it, taken through W_v (src/attention.c:812-815): grid (heads,
// 2), 512 threads. A block merges 256 of its head's 512 columns, two threads a column (each half of the records), and forms
// those columns' part of the head's 128 values, eight per warp, whose weights are on their way before the records are
// there; attn [2][heads][128] has the two parts, added up by the next projection. The kernel is one block per SM and trips to L2, so
// where the records are more than 32 a thread asks for 36 at once, all of its half for 9216 rows: a call over 8191 rows 84 -> 75 us
// (16 at a time for every number, in registers for two blocks that there never are; at 1000 rows, 8 records, 16 are 1 us ahead).
template <int AHEAD>
__global__ void __launch_bounds__(512, AHEAD > 16 ? 1 : 2) merge_unabsorb_kernel(const float *partial, int nsplit, int nh, const uint16_t *kvb, int nope, float *attn) {
    constexpr int L = 512, VD = 128;
    __shared__ float s_w[512], s_red[32], s_half[256];
    __shared__ __align__(16) float s_c[256];
    const int h = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, c0 = blockIdx.y * 256;
    const int64_t rec = (int64_t)nh * (L + 2);
    cwk_pdl_launch();
    uint4 v[8];
#pragma unroll
    for (int r = 0; r < 8; r++) v[r] = ld_weight16(kvb + ((int64_t)h * (nope + VD) + nope + warp * 8 + r) * L + c0 + lane * 8);
    cwk_pdl_wait();
    const int lo = tid < 256 ? 0 : (nsplit + 1) / 2, hi = tid < 256 ? (nsplit + 1) / 2 : nsplit;      // this thread's records
    const float *col = partial + 2 * nh + (int64_t)h * L + c0 + (tid & 255);
    float o[AHEAD];
#pragma unroll
    for (int s = 0; s < AHEAD; s++) o[s] = lo + s < hi ? col[(lo + s) * rec] : 0.f;
    float m = -INFINITY, l = 0.f;                          // record `tid`
    if (tid < nsplit) {
        const float mm = partial[tid * rec + h];
        l = partial[tid * rec + nh + h];
        if (l > 0.f) m = mm;
    }
    float M = m;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, d));
    if (lane == 0) s_red[warp] = M;
    __syncthreads();
    M = s_red[lane & 15];
#pragma unroll
    for (int d = 8; d > 0; d >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, d));
    const float w = m == -INFINITY ? 0.f : __expf(m - M);
    float den = w * l;
    s_w[tid] = w;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) den += __shfl_xor_sync(0xffffffffu, den, d);
    if (lane == 0) s_red[16 + warp] = den;
    __syncthreads();
    den = s_red[16 + (lane & 15)];
#pragma unroll
    for (int d = 8; d > 0; d >>= 1) den += __shfl_xor_sync(0xffffffffu, den, d);
    float a[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int s = 0; s < AHEAD; s++)
        if (lo + s < hi) a[s & 3] += s_w[lo + s] * o[s];
    for (int s0 = lo + AHEAD; s0 < hi; s0 += AHEAD) {
#pragma unroll
        for (int s = 0; s < AHEAD; s++) o[s] = s0 + s < hi ? col[(s0 + s) * rec] : 0.f;
#pragma unroll
        for (int s = 0; s < AHEAD; s++)
            if (s0 + s < hi) a[s & 3] += s_w[s0 + s] * o[s];
    }
    const float sum = (a[0] + a[1]) + (a[2] + a[3]), inv = den > 0.f ? 1.f / den : 0.f;
    if (tid >= 256) s_half[tid - 256] = sum;
    __syncthreads();
    if (tid < 256) s_c[tid] = __uint_as_float(pack_bf16x2(0.f, (sum + s_half[tid]) * inv) & 0xffff0000u);
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 8; r++) {
        float t = gemv_piece<GEMV_BF16>(v[r], s_c, lane * 8, nullptr);
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) t += __shfl_xor_sync(0xffffffffu, t, d);
        if (lane == 0) attn[((int64_t)blockIdx.y * nh + h) * VD + warp * 8 + r] = t;
    }
}
