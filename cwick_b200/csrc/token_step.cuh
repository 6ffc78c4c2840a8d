// token_step.cuh -- kernels of the reference-named decode call for one token (src/attention.c:642-902), included by dropin.cu
// behind its projection helpers.
//
// A token's projections are their weights read once: 126 MB in BF16 for a layer of hidden 4096, 19 us of HBM time. What a
// chain of eight kernels adds to that is latency -- a kernel comes up, asks for its first bytes, waits a microsecond, and at
// its end HBM idles until the next one has done the same (100 us per call). So here every kernel (1) comes up while the one
// before still runs (cwk_launch_early) and asks for its first weights, which depend on nothing, before it waits for its
// activations; (2) the first projection and the attention, which leave HBM idle, tell L2 to fetch the weights that are next
// (`Prefetch`); and (3) small steps ride along: the two norms in the q_b projection's blocks, the merge of the attention's
// split records in the un-absorb.
#pragma once

struct Prefetch {               // a range to bring into L2, dealt out to a grid's blocks
    const void *p;
    size_t bytes;
};
// One thread of every block; 16-byte units, at most 64 KB per instruction.
__device__ __forceinline__ void prefetch_share(const Prefetch &f, int block, int blocks) {
    if (!f.bytes) return;
    const size_t share = ((f.bytes + blocks - 1) / blocks + 15) & ~(size_t)15;
    size_t at = (size_t)block * share;
    const size_t end = at + share < f.bytes ? at + share : (f.bytes & ~(size_t)15);
    while (at < end) {
        const uint32_t n = (uint32_t)(end - at < 65536 ? end - at : 65536);
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"((const uint8_t *)f.p + at), "r"(n) : "memory");
        at += n;
    }
}

// y[r] = W[r] . x for one token (as gemv_rows_kernel, rows of whole 16-byte pieces only). NORM: x is first normalised,
// x / sqrt(mean(x^2) + eps) * w, by every block for itself (its values in shared memory, the sum in rms_scale_row's order);
// the launch's last block then is not a projection block but does the kv_a row: normalised in place, narrowed into the
// cache row and written to the caller's staging.
struct TokenNorm {
    const uint16_t *w, *wkv;
    float eps;
    float *kva;
    int nkv;
    uint16_t *row_out;
    void *host_row;
    int host_bf16;
};
template <int KIND, bool NORM>
__global__ void __launch_bounds__(256) gemv_token_kernel(const void *Wv, const float *scales, const float *x, float *y, int rows, int k, int rpb, int nb1,
                                                         const void *W2, const float *scales2, float *y2, int rows2, const TokenNorm nm, const Prefetch f0,
                                                         const Prefetch f1) {
    constexpr int E = KIND == GEMV_BF16 ? 8 : KIND == GEMV_F32 ? 4 : 16, EB = 16 / E, AHEAD = 8;
    extern __shared__ __align__(16) float s_x[];
    __shared__ float s_part[8];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    cwk_pdl_launch();
    if (NORM && blockIdx.x == gridDim.x - 1) {
        cwk_pdl_wait();
        rms_scale_row(nm.kva, nm.nkv, nm.wkv, nm.eps, nm.row_out, nm.host_row, nm.host_bf16);
        return;
    }
    const int wpr = 8 / rpb;                               // warps per row
    int bx = blockIdx.x;
    if (bx >= nb1) { bx -= nb1; Wv = W2; scales = scales2; y = y2; rows = rows2; }
    const int r = bx * rpb + warp / wpr, part = warp % wpr;
    const bool live = r < rows;
    const uint8_t *w = reinterpret_cast<const uint8_t *>(Wv) + (int64_t)(live ? r : 0) * k * EB;
    const float *sc = KIND == GEMV_FP8 ? scales + (int64_t)((live ? r : 0) / 128) * ((k + 127) / 128) : nullptr;
    const int step = wpr * 32 * E, j0 = (part * 32 + lane) * E;
    uint4 v[AHEAD];
#pragma unroll
    for (int u = 0; u < AHEAD; u++)
        if (j0 + u * step < k) v[u] = ld_weight16(w + (int64_t)(j0 + u * step) * EB);
    if ((lane & 7) == 0)                                   // the row's further lines on their way to L2
        for (int j = j0 + AHEAD * step; j < k; j += step) asm volatile("prefetch.global.L2 [%0];" ::"l"(w + (int64_t)j * EB));
    if (threadIdx.x == 0) {
        prefetch_share(f0, blockIdx.x, gridDim.x);
        prefetch_share(f1, blockIdx.x, gridDim.x);
    }
    cwk_pdl_wait();
    if (NORM) {
        for (int i = threadIdx.x; i < k; i += 256) s_x[i] = x[i];      // (each thread scales what it read)
        rms_scale_row(s_x, k, nm.w, nm.eps, nullptr, nullptr, 0);
        __syncthreads();
        x = s_x;
    }
    float acc = 0.f;
    int j = j0;
#pragma unroll
    for (int u = 0; u < AHEAD; u++)
        if (j0 + u * step < k) acc += gemv_piece<KIND>(v[u], x, j0 + u * step, sc);
    for (j = j0 + AHEAD * step; j + (AHEAD - 1) * step < k; j += AHEAD * step) {
#pragma unroll
        for (int u = 0; u < AHEAD; u++) v[u] = ld_weight16(w + (int64_t)(j + u * step) * EB);
#pragma unroll
        for (int u = 0; u < AHEAD; u++) acc += gemv_piece<KIND>(v[u], x, j + u * step, sc);
    }
    for (; j < k; j += step) acc += gemv_piece<KIND>(ld_weight16(w + (int64_t)j * EB), x, j, sc);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (wpr == 1) {
        if (lane == 0 && live) y[r] = acc;
        return;
    }
    if (lane == 0) s_part[warp] = acc;
    __syncthreads();
    if (part == 0 && lane == 0 && live) {
        float sum = 0.f;
        for (int i = 0; i < wpr; i++) sum += s_part[warp + i];
        y[r] = sum;
    }
}
bool gemv_token_ok(const WeightMirror *w, const void *x) {
    const int E = w->kind == CWKC_WEIGHT_BF16 ? 8 : w->kind == CWKC_WEIGHT_F32 ? 4 : 16;
    return w->cols % E == 0 && ((reinterpret_cast<uintptr_t>(w->data) | reinterpret_cast<uintptr_t>(x)) & 15) == 0 && w->rows < (1 << 30);
}
// w2 != NULL: a second matrix of the same kind and width, in the same launch. norm != NULL: NORM (no second matrix).
cudaError_t gemv_token(cwk_ctx *ctx, const WeightMirror *w, const float *x, float *y, const WeightMirror *w2, float *y2, const TokenNorm *norm, Prefetch f0, Prefetch f1) {
    int rpb = 8;                                           // fewer rows per block until the grid is a few blocks per SM
    const int64_t rows2 = w2 ? w2->rows : 0;
    while (rpb > 1 && (w->rows + rpb - 1) / rpb + (rows2 + rpb - 1) / rpb < 4 * (int64_t)ctx->sm_count) rpb >>= 1;
    const int nb1 = (int)((w->rows + rpb - 1) / rpb), nb2 = (int)((rows2 + rpb - 1) / rpb);
    const TokenNorm nm = norm ? *norm : TokenNorm{};
    auto go = [&](auto kern) {
        ctx->launches++;
        return cwk_launch_early(kern, dim3((unsigned)(nb1 + nb2 + (norm ? 1 : 0))), dim3(256), norm ? (size_t)w->cols * 4 : 0, ctx->stream, (const void *)w->data, (const float *)w->scales, x, y,
                                (int)w->rows, (int)w->cols, rpb, nb1, (const void *)(w2 ? w2->data : nullptr), (const float *)(w2 ? w2->scales : nullptr), y2, (int)rows2, nm, f0, f1);
    };
    if (w->kind == CWKC_WEIGHT_BF16) return norm ? go(gemv_token_kernel<GEMV_BF16, true>) : go(gemv_token_kernel<GEMV_BF16, false>);
    if (w->kind == CWKC_WEIGHT_F32) return norm ? go(gemv_token_kernel<GEMV_F32, true>) : go(gemv_token_kernel<GEMV_F32, false>);
    return norm ? go(gemv_token_kernel<GEMV_FP8, true>) : go(gemv_token_kernel<GEMV_FP8, false>);
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

// The attention's split records of one token (nsplit x [heads][512 + 2], flash_rows.cuh's layout) merged, and the result,
// rounded to bf16 as the merge on its own would leave it, taken through W_v (src/attention.c:812-815): grid (heads, 2),
// 512 threads; a block merges its head's 512 columns and does half of the head's 128 value rows, four per warp, whose weights
// are on their way before the records are there.
__global__ void __launch_bounds__(512) merge_unabsorb_kernel(const float *partial, int nsplit, int nh, const uint16_t *kvb, int nope, float *attn) {
    constexpr int L = 512, VD = 128, AHEAD = 32;
    __shared__ float s_w[512], s_red[32];
    __shared__ __align__(16) float s_c[L];
    const int h = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int64_t rec = (int64_t)nh * (L + 2);
    cwk_pdl_launch();
    uint4 v[4][2];
    const int r0 = blockIdx.y * (VD / 2) + warp * 4;
#pragma unroll
    for (int r = 0; r < 4; r++) {
        const uint16_t *w = kvb + ((int64_t)h * (nope + VD) + nope + r0 + r) * L;
        v[r][0] = ld_weight16(w + lane * 8);
        v[r][1] = ld_weight16(w + 256 + lane * 8);
    }
    cwk_pdl_wait();
    const float *col = partial + 2 * nh + (int64_t)h * L + tid;
    float o[AHEAD];
#pragma unroll
    for (int s = 0; s < AHEAD; s++) o[s] = s < nsplit ? col[s * rec] : 0.f;
    float m = -INFINITY, l = 0.f;                          // this thread's record (nsplit <= 512)
    if (tid < nsplit) {
        l = partial[tid * rec + nh + h];
        if (l > 0.f) m = partial[tid * rec + h];
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
        if (s < nsplit) a[s & 3] += s_w[s] * o[s];
    for (int s0 = AHEAD; s0 < nsplit; s0 += AHEAD) {
#pragma unroll
        for (int s = 0; s < AHEAD; s++) o[s] = s0 + s < nsplit ? col[(s0 + s) * rec] : 0.f;
#pragma unroll
        for (int s = 0; s < AHEAD; s++)
            if (s0 + s < nsplit) a[s & 3] += s_w[s0 + s] * o[s];
    }
    const float inv = den > 0.f ? 1.f / den : 0.f;
    s_c[tid] = __uint_as_float(pack_bf16x2(0.f, ((a[0] + a[1]) + (a[2] + a[3])) * inv) & 0xffff0000u);
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 4; r++) {
        float t = gemv_piece<GEMV_BF16>(v[r][0], s_c, lane * 8, nullptr) + gemv_piece<GEMV_BF16>(v[r][1], s_c, 256 + lane * 8, nullptr);
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) t += __shfl_xor_sync(0xffffffffu, t, d);
        if (lane == 0) attn[h * VD + r0 + r] = t;
    }
}
