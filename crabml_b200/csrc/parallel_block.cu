// parallel_block.cu -- the two products of a layer whose sublayers stand side by side on one norm, each fused with what surrounds it:
//
//   cc_layer_norm_product        out = W LN(x): the norm is taken while the product's operand is made, so the normed rows never exist in memory
//                                as 32-bit floats.
//   cc_joined_product_accumulate x += [W_a | W_b] [a ; glu(g, u)]: the output projections of mixer and feed-forward as ONE product over the
//                                mixer's result and the gated units, which are computed while the operand is made; the residual sum is the
//                                product's epilogue.
//
// Three forms, chosen like those of the plain product (dense.cu):
//   fewer than 8 rows            pb_matvec_kernel: every CTA stages the operand row in shared memory (norm or gated units included) and streams
//                                its weight rows past it
//   BF16, 32 rows or more, columns a multiple of 64: a kernel writes the bfloat16 operand straight from the 32-bit inputs, then the tensor-core product
//   everything else              a 32-bit operand in scratch, then the SIMT tiles
// BF16 matrices: the operand is rounded to bfloat16 once, products are exact, sums are 32-bit; F32 matrices: everything is 32-bit.
#include <cuda_bf16.h>

#include "../../include/crabml_seqops.h"
#include "act.cuh"
#include "capi_checks.cuh"
#include "layer_norm.cuh"

bool cc_prefill_bf16_supported(int64_t m, int64_t k, int64_t b);                                                                                              // prefill_gemm.cu
int cc_prefill_bf16_operand(cc_device* dev, int64_t b, int64_t k, void** out);
int cc_launch_prefill_bf16_operand(cc_device* dev, const cc_buf* w, float* out, int64_t m, int64_t k, int64_t b, int accumulate);
int cc_launch_dense_tile(cc_device* dev, const cc_buf* w, const float* x, float* out, int64_t m, int64_t k, int64_t b, int accumulate);                        // dense.cu

#define PB_COLS 1024                       // columns of the operand that a warp holds, 32 a lane
#define PB_TURNS 32                        // rows of a warp whose sums wait in shared memory
#define PB_DEPTH 4                         // 16-byte pieces of a weight row that a lane has in flight where the operand stays in shared memory
#define PB_LN_THREADS 256

// what the operand's rows are made of
struct PbNorm {
    const float *x, *w, *b;                // x: [T, k] contiguous; b NULL: no bias
    float eps;
    static constexpr bool NORM = true;
    template <int THREADS, int EACH>
    __device__ __forceinline__ void stage(float* dst, int t, int k, float* red, bool round) const {
        layer_norm_row<THREADS>(x + (int64_t)t * k, w, b, k, eps, red, [&](int c, float v) { dst[c] = round ? __bfloat162float(__float2bfloat16_rn(v)) : v; });
    }
};
struct PbJoin {
    const float *a, *g, *u;                // a: [T, ca] contiguous; g, u: gate and up numbers of row t at g + t * rs, u + t * rs
    int64_t rs;
    int ca, ff;
    cc_glu_params P;
    __device__ __forceinline__ float at(int t, int c) const {
        return c < ca ? a[(int64_t)t * ca + c] : glu_apply(g[t * rs + (c - ca)], u[t * rs + (c - ca)], P);
    }
    static constexpr bool NORM = false;
    template <int THREADS, int EACH>
    __device__ __forceinline__ void stage(float* dst, int t, int k, float*, bool round) const {
        if constexpr (EACH == 1) {
            for (int c = threadIdx.x; c < k; c += THREADS) {
                const float v = at(t, c);
                dst[c] = round ? __bfloat162float(__float2bfloat16_rn(v)) : v;
            }
            return;
        }
        for (int c0 = threadIdx.x; c0 < k; c0 += EACH * THREADS) {       // the numbers of EACH columns at once
            float x[EACH], y[EACH];
#pragma unroll
            for (int e = 0; e < EACH; e++) {
                const int c = c0 + e * THREADS;
                x[e] = y[e] = 0.0f;
                if (c < ca) x[e] = a[(int64_t)t * ca + c];
                else if (c < k) { x[e] = g[t * rs + (c - ca)]; y[e] = u[t * rs + (c - ca)]; }
            }
#pragma unroll
            for (int e = 0; e < EACH; e++) {
                const int c = c0 + e * THREADS;
                const float v = c < ca ? x[e] : glu_apply(x[e], y[e], P);
                if (c < k) dst[c] = round ? __bfloat162float(__float2bfloat16_rn(v)) : v;
            }
        }
    }
};

// grid (about one CTA per SM, T).  `split` warps (a power of two) share one weight row, each a contiguous stretch of its 16-byte pieces, PB_COLS columns or less at a time;
// a CTA owns WARPS / split rows at a time.  A lane holds its 32 columns of the operand in registers for all of the warp's rows and has the pieces of the
// next row in flight while it multiplies those of this one; the first are fetched before the operand row is staged.  Sums of a row: each piece by itself, the pieces, the
// butterfly, then the row's warps in ascending order, once for up to PB_TURNS rows.  The order depends on the sizes alone, not on T.
// Bound by latency (norm, first pieces) and, in a model's head, by memory.  With the operand read from shared memory for every row, 32 warps took 4096 cycles of its ports for
// 64 rows of 1024 columns (lanes 32 bytes apart: two turns each).  What both kernels measured, and where the line between them lies: pb_launch_matvec.
template <bool BF16W, class Op, int THREADS>
__global__ void __launch_bounds__(THREADS, 1) pb_matvec_kernel(const void* __restrict__ W, Op op, float* __restrict__ out, int m, int k, int split, int accumulate) {
    extern __shared__ __align__(16) float pb_sm[];              // the operand row, k floats (rounded up to 4)
    constexpr int WARPS = THREADS / 32;
    __shared__ float red[WARPS], part[PB_TURNS][WARPS];
    constexpr bool AHEAD = THREADS <= 512;                       // registers for the next row's pieces
    constexpr int PIECE = BF16W ? 8 : 4, DEPTH = PB_COLS / 32 / PIECE;      // columns of a piece ; pieces a lane holds
    const int t = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int per_cta = WARPS / split, sub = warp % split, slot = warp / split;
    const int rows_it = (m + gridDim.x * per_cta - 1) / (gridDim.x * per_cta);
    const int row0 = blockIdx.x * per_cta + slot, row_step = gridDim.x * per_cta;
    float* orow = out + (int64_t)t * m;
    const bool vec = k % PIECE == 0;
    const int pieces = k / PIECE, per_warp = (pieces + split - 1) / split;
    const int p_begin = min(pieces, sub * per_warp), p_end = min(pieces, p_begin + per_warp), blocks = vec ? (per_warp + 32 * DEPTH - 1) / (32 * DEPTH) : 1;
    int4 cur[DEPTH], nxt[AHEAD ? DEPTH : 1];
    auto fetch = [&](int4 (&v)[DEPTH], int it, int b) {
        const int p0 = p_begin + b * 32 * DEPTH + lane, row = row0 + it * row_step;
#pragma unroll
        for (int e = 0; e < DEPTH; e++) {
            const int p = p0 + e * 32;
            v[e] = (row < m && p < p_end) ? ld_stream_16((const uint8_t*)W + ((int64_t)row * pieces + p) * 16) : make_int4(0, 0, 0, 0);
        }
    };
    // this CTA's weight rows start for L2 while the kernel before is still at work (a prefetch has no value that could be stale): with the rows of 15 MB
    // fetched only behind the norm, the product took 12.8 us for 2.3 us of memory time
    if (blockIdx.y == 0) {
        const unsigned row_bytes = (unsigned)k * (BF16W ? 2 : 4), lines = (row_bytes + 127) >> 7;
        for (int it = 0; it < rows_it; it++)
            for (unsigned i = threadIdx.x; i < per_cta * lines; i += THREADS) {
                const unsigned r = i / lines;
                const int64_t row = blockIdx.x * per_cta + (int64_t)it * row_step + r;
                if (row < m) asm volatile("prefetch.global.L2 [%0];" ::"l"((const uint8_t*)W + row * row_bytes + ((i - r * lines) << 7)));
            }
    }
    pdl_enter();
    if (vec) fetch(cur, 0, 0);
    op.template stage<THREADS, 4>(pb_sm, t, k, red, BF16W);
    __syncthreads();
    for (int it0 = 0; it0 < rows_it; it0 += PB_TURNS) {
        const int turns = min(PB_TURNS, rows_it - it0);
        for (int b = 0; b < blocks; b++) {
            float x[PB_COLS / 32];
#pragma unroll
            for (int e = 0; e < DEPTH; e++) {
                const int p = p_begin + b * 32 * DEPTH + lane + e * 32;
                const bool in = vec && p < p_end;
#pragma unroll
                for (int c = 0; c < PIECE; c += 4) {
                    const float4 v = in ? *(const float4*)(pb_sm + p * PIECE + c) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    x[e * PIECE + c] = v.x; x[e * PIECE + c + 1] = v.y; x[e * PIECE + c + 2] = v.z; x[e * PIECE + c + 3] = v.w;
                }
            }
            for (int it = 0; it < turns; it++) {
                float acc = 0.0f;
                if (vec) {
                    const bool more = it + 1 < turns;             // the next row of this block, or the first one of the next
                    const int nb = more ? b : b + 1 < blocks ? b + 1 : 0, ni = more ? it0 + it + 1 : b + 1 < blocks ? it0 : it0 + PB_TURNS;
                    if constexpr (AHEAD) { if (ni < rows_it) fetch(nxt, ni, nb); }
                    float piece[DEPTH];
#pragma unroll
                    for (int e = 0; e < DEPTH; e++) {
                        const float* y = x + e * PIECE;
                        float a = 0.0f;
                        if (BF16W) {
                            a = fmaf(__uint_as_float((unsigned)cur[e].x << 16), y[0], a); a = fmaf(__uint_as_float((unsigned)cur[e].x & 0xFFFF0000u), y[1], a);
                            a = fmaf(__uint_as_float((unsigned)cur[e].y << 16), y[2], a); a = fmaf(__uint_as_float((unsigned)cur[e].y & 0xFFFF0000u), y[3], a);
                            a = fmaf(__uint_as_float((unsigned)cur[e].z << 16), y[4 % PIECE], a); a = fmaf(__uint_as_float((unsigned)cur[e].z & 0xFFFF0000u), y[5 % PIECE], a);
                            a = fmaf(__uint_as_float((unsigned)cur[e].w << 16), y[6 % PIECE], a); a = fmaf(__uint_as_float((unsigned)cur[e].w & 0xFFFF0000u), y[7 % PIECE], a);
                        } else {
                            a = fmaf(__int_as_float(cur[e].x), y[0], a); a = fmaf(__int_as_float(cur[e].y), y[1], a);
                            a = fmaf(__int_as_float(cur[e].z), y[2], a); a = fmaf(__int_as_float(cur[e].w), y[3], a);
                        }
                        piece[e] = a;
                    }
#pragma unroll
                    for (int n = DEPTH / 2; n >= 1; n /= 2)
#pragma unroll
                        for (int e = 0; e < n; e++) piece[e] += piece[e + n];
                    acc = piece[0];
                    if constexpr (AHEAD) {
#pragma unroll
                        for (int e = 0; e < DEPTH; e++) cur[e] = nxt[e];
                    } else if (ni < rows_it) fetch(cur, ni, nb);
                } else {
                    const int row = row0 + (it0 + it) * row_step;
                    if (row < m)
                        for (int c = sub * 32 + lane; c < k; c += split * 32)
                            acc = fmaf(BF16W ? __uint_as_float((unsigned)((const uint16_t*)W)[(int64_t)row * k + c] << 16) : ((const float*)W)[(int64_t)row * k + c], pb_sm[c], acc);
                }
                acc = warp_sum(acc);
                if (lane == 0) part[it][warp] = b ? part[it][warp] + acc : acc;
            }
        }
        __syncthreads();
        for (int i = threadIdx.x; i < turns * per_cta; i += THREADS) {
            const int it = i / per_cta, r = i - it * per_cta, row = blockIdx.x * per_cta + r + (it0 + it) * row_step;
            float a = 0.0f;
            for (int y = 0; y < split; y++) a += part[it][r * split + y];
            if (row < m) orow[row] = accumulate ? orow[row] + a : a;
        }
        if (it0 + PB_TURNS < rows_it) __syncthreads();            // part is written again
    }
}
__device__ __forceinline__ float pb_dot8(const int4 v, const float* a, float acc) {
    const float4 a0 = *(const float4*)a, a1 = *(const float4*)(a + 4);
    acc = fmaf(__uint_as_float((unsigned)v.x << 16), a0.x, acc); acc = fmaf(__uint_as_float((unsigned)v.x & 0xFFFF0000u), a0.y, acc);
    acc = fmaf(__uint_as_float((unsigned)v.y << 16), a0.z, acc); acc = fmaf(__uint_as_float((unsigned)v.y & 0xFFFF0000u), a0.w, acc);
    acc = fmaf(__uint_as_float((unsigned)v.z << 16), a1.x, acc); acc = fmaf(__uint_as_float((unsigned)v.z & 0xFFFF0000u), a1.y, acc);
    acc = fmaf(__uint_as_float((unsigned)v.w << 16), a1.z, acc); acc = fmaf(__uint_as_float((unsigned)v.w & 0xFFFF0000u), a1.w, acc);
    return acc;
}
// The same with the operand row in shared memory, where one batch of PB_DEPTH pieces a lane is all of a warp's part or a CTA has few rows (pb_launch_matvec): half the
// registers, 32 warps, a sum of one chain.  `split` warps share a row, each a contiguous stretch of its pieces in lane-strided order; a lane keeps the next pieces -- of
// this row or of the next one -- in flight while it multiplies the current ones.  Partial sums: the butterfly, then the row's warps in ascending order.
template <bool BF16W, class Op>
__global__ void __launch_bounds__(1024, 1) pb_matvec_shared_kernel(const void* __restrict__ W, Op op, float* __restrict__ out, int m, int k, int split, int accumulate) {
    extern __shared__ __align__(16) float pb_sm[];              // the operand row, k floats (rounded up to 4)
    __shared__ float red[32];
    const int t = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int per_cta = 32 / split, sub = warp % split, slot = warp / split;
    const int rows_it = (m + gridDim.x * per_cta - 1) / (gridDim.x * per_cta);
    const int row0 = blockIdx.x * per_cta + slot, row_step = gridDim.x * per_cta;
    float* orow = out + (int64_t)t * m;
    const bool vec = BF16W ? (k & 7) == 0 : (k & 3) == 0;
    const int pieces = BF16W ? k >> 3 : k >> 2;                  // 16-byte pieces of a row
    const int per_warp = (pieces + split - 1) / split;
    const int p_begin = min(pieces, sub * per_warp), p_end = min(pieces, p_begin + per_warp);
    const int batches = (per_warp + 32 * PB_DEPTH - 1) / (32 * PB_DEPTH);
    const int total = rows_it * batches;
    int4 cur[PB_DEPTH], nxt[PB_DEPTH];
    auto fetch = [&](int4* v, int i) {
        const int it = i / batches, p0 = p_begin + (i - it * batches) * 32 * PB_DEPTH + lane;
        const int row = row0 + it * row_step;
#pragma unroll
        for (int e = 0; e < PB_DEPTH; e++) {
            const int p = p0 + e * 32;
            v[e] = (row < m && p < p_end) ? ld_stream_16((const uint8_t*)W + ((int64_t)row * pieces + p) * 16) : make_int4(0, 0, 0, 0);
        }
    };
    // this CTA's weight rows start for L2 while the kernel before is still at work (a prefetch has no value that could be stale): with the rows of 15 MB
    // fetched only behind the norm, the product took 12.8 us for 2.3 us of memory time
    {
        const int64_t row_bytes = (int64_t)k * (BF16W ? 2 : 4);
        for (int64_t i = threadIdx.x; i < (int64_t)rows_it * per_cta * ((row_bytes + 127) >> 7); i += 1024) {
            const int64_t r = i / ((row_bytes + 127) >> 7), at = (i - r * ((row_bytes + 127) >> 7)) << 7, row = blockIdx.x * per_cta + (r / per_cta) * row_step + r % per_cta;
            if (row < m && blockIdx.y == 0) asm volatile("prefetch.global.L2 [%0];" ::"l"((const uint8_t*)W + row * row_bytes + at));
        }
    }
    pdl_enter();
    if (vec) fetch(cur, 0);
    op.template stage<1024, 1>(pb_sm, t, k, red, BF16W);
    __syncthreads();
    for (int it = 0; it < rows_it; it++) {
        const int row = row0 + it * row_step;
        float acc = 0.0f;
        if (vec) {
            for (int b = 0; b < batches; b++) {
                const int i = it * batches + b;
                if (i + 1 < total) fetch(nxt, i + 1);
                const int p0 = p_begin + b * 32 * PB_DEPTH + lane;
#pragma unroll
                for (int e = 0; e < PB_DEPTH; e++) {
                    const int p = p0 + e * 32;
                    if (p < p_end) {
                        if (BF16W) acc = pb_dot8(cur[e], pb_sm + p * 8, acc);
                        else {
                            const float4 a = *(const float4*)(pb_sm + p * 4);
                            acc = fmaf(__int_as_float(cur[e].x), a.x, acc); acc = fmaf(__int_as_float(cur[e].y), a.y, acc);
                            acc = fmaf(__int_as_float(cur[e].z), a.z, acc); acc = fmaf(__int_as_float(cur[e].w), a.w, acc);
                        }
                    }
                }
#pragma unroll
                for (int e = 0; e < PB_DEPTH; e++) cur[e] = nxt[e];
            }
        } else if (row < m) {
            for (int c = sub * 32 + lane; c < k; c += split * 32)
                acc = fmaf(BF16W ? __uint_as_float((unsigned)((const uint16_t*)W)[(int64_t)row * k + c] << 16) : ((const float*)W)[(int64_t)row * k + c], pb_sm[c], acc);
        }
        acc = warp_sum(acc);
        if (split > 1) {
            __syncthreads();                                     // red may still be read
            if (lane == 0) red[warp] = acc;
            __syncthreads();
            if (sub == 0) {
                acc = 0.0f;
                for (int s = 0; s < split; s++) acc += red[warp + s];
            }
        }
        if (lane == 0 && sub == 0 && row < m) orow[row] = accumulate ? orow[row] + acc : acc;
    }
}
// the bfloat16 operand of the tensor-core product: a CTA per row
__global__ void __launch_bounds__(PB_LN_THREADS) pb_norm_bf16_kernel(const float* __restrict__ x, const float* __restrict__ w, const float* __restrict__ b, __nv_bfloat16* __restrict__ out,
                                                                     int k, float eps) {
    pdl_enter();
    __shared__ float red[PB_LN_THREADS / 32];
    __nv_bfloat16* o = out + (int64_t)blockIdx.x * k;
    layer_norm_row<PB_LN_THREADS>(x + (int64_t)blockIdx.x * k, w, b, k, eps, red, [&](int c, float v) { o[c] = __float2bfloat16_rn(v); });
}
__global__ void __launch_bounds__(PB_LN_THREADS) pb_norm_f32_kernel(const float* __restrict__ x, const float* __restrict__ w, const float* __restrict__ b, float* __restrict__ out, int k,
                                                                    float eps) {
    pdl_enter();
    __shared__ float red[PB_LN_THREADS / 32];
    float* o = out + (int64_t)blockIdx.x * k;
    layer_norm_row<PB_LN_THREADS>(x + (int64_t)blockIdx.x * k, w, b, k, eps, red, [&](int c, float v) { o[c] = v; });
}
// grid (columns / 512, rows): two neighbouring columns per thread; k is even
__global__ void __launch_bounds__(256) pb_join_bf16_kernel(PbJoin op, __nv_bfloat16* __restrict__ out, int k) {
    pdl_enter();
    const int c = (blockIdx.x * 256 + threadIdx.x) * 2, t = blockIdx.y;
    if (c < k) *(__nv_bfloat162*)(out + (int64_t)t * k + c) = __floats2bfloat162_rn(op.at(t, c), op.at(t, c + 1));
}
// the same, 8 neighbouring columns per thread, where both parts and the rows of all operands are whole pieces of 16 bytes (SWISH: units known to
// be that, without the code of the others).
// grid (columns / 1024, rows).  512 x (1024 + 3072), us: two columns a thread, any unit 6.6 ; here 4.9 (509 x (2048 + 6144): 11.4, 6.4)
template <bool SWISH>
__global__ void __launch_bounds__(128) pb_join8_bf16_kernel(PbJoin op, __nv_bfloat16* __restrict__ out, int k) {
    pdl_enter();
    const int c = (blockIdx.x * 128 + threadIdx.x) * 8, t = blockIdx.y;
    if (c >= k) return;
    float v[8];
    if (c < op.ca) {
        const float* a = op.a + (int64_t)t * op.ca + c;
        *(float4*)v = *(const float4*)a; *(float4*)(v + 4) = *(const float4*)(a + 4);
    } else {
        const float *gp = op.g + t * op.rs + (c - op.ca), *up = op.u + t * op.rs + (c - op.ca);
        float g[8], u[8];
        *(float4*)g = *(const float4*)gp; *(float4*)(g + 4) = *(const float4*)(gp + 4);
        *(float4*)u = *(const float4*)up; *(float4*)(u + 4) = *(const float4*)(up + 4);
        cc_glu_params P = op.P;
        if (SWISH) P.act = CC_ACT_SWISH;
#pragma unroll
        for (int e = 0; e < 8; e++) v[e] = glu_apply(g[e], u[e], P);
    }
    __nv_bfloat162 o[4];
#pragma unroll
    for (int e = 0; e < 4; e++) o[e] = __floats2bfloat162_rn(v[2 * e], v[2 * e + 1]);
    *(uint4*)(out + (int64_t)t * k + c) = *(const uint4*)o;
}
__global__ void __launch_bounds__(256) pb_join_f32_kernel(PbJoin op, float* __restrict__ out, int k) {
    pdl_enter();
    const int c = blockIdx.x * 256 + threadIdx.x, t = blockIdx.y;
    if (c < k) out[(int64_t)t * k + c] = op.at(t, c);
}

static const size_t PB_MAX_SMEM = 200 * 1024;
static bool pb_few(int64_t T, int64_t k) { return T < 8 && (size_t)((k + 3) & ~3) * 4 <= PB_MAX_SMEM; }
template <class Op>
static int pb_launch_matvec_by(cc_device* dev, void (*kernel)(const void*, Op, float*, int, int, int, int), int threads, const cc_buf* w, const Op& op, float* out, int64_t m, int64_t k, int64_t T,
                               int accumulate, int split) {
    const size_t smem = (size_t)((k + 3) & ~3) * 4;
    if (smem > 40 * 1024) CC_CUDA(dev, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    // one CTA fits an SM, and staging the operand is most of a short call: the T rows share the SMs, so that no SM stages twice.  us with all SMs for each row / here,
    // 7424 x 1024 behind the norm: 2 rows 13.1 / 9.8, 7 rows 41 / 20 ; 1024 x 4096 behind the gated units: 10.8 / 7.1, 33 / 12
    const int64_t per_cta = threads / 32 / split, need = (m + per_cta - 1) / per_cta, ctas = dev->sm_count / T < 1 ? 1 : dev->sm_count / T;
    cc_launch_pdl(dev, kernel, dim3((unsigned)(need < ctas ? need : ctas), (unsigned)T), threads, smem, w->plane[0], op, out, (int)m, (int)k, split, accumulate);
    CC_LAUNCH_CHECK(dev);
    return CC_OK;
}
// Which kernel follows from the sizes and the weights' type alone, so that a row has the same bits in every call.  us of one row, operand in shared memory with 32 warps /
// in registers with 16 / in registers with 32:
//   norm, bfloat16    2000 x 384 5.2 / 4.0 / 5.9 ; 7424 x 1024 9.5 / 7.6 / 8.6 ; 18432 x 1024 15.4 / 12.5 / 12.4 ; 32000 x 1024 23.3 / 18.1 / 16.7 ; 6000 x 2048 13.1 / 10.1 / 10.5 ;
//                     12288 x 2048 18.2 / 15.1 / 14.8 ; 32000 x 1536 28.5 / 31.2 / 24.4 ; 18432 x 3072 30.1 / 35.6 / 27.1: 16 warps stage sooner, 32 ask for more at a time
//   norm, 32 bits     4000 x 512 5.7 / 5.4 ; 12288 x 512 9.3 / 9.3 ; 32000 x 512 16.0 / 16.9 ; 7424 x 1024 10.3 / 9.3 ; 32000 x 1024 25.7 / 23.6 ; 32000 x 1536 35.8 / 36.9  (32 warps spill)
//   units, bfloat16   512 x 2048 4.4 / 4.0 / 4.7 ; 768 x 3072 5.4 / 6.4 / 5.7 ; 1024 x 4096 6.6 / 6.6 / 6.2 ; 1280 x 7680 12.4 / 11.9 / 10.5 ; 1536 x 9216 14.4 / 18.0 / 15.1 ;
//                     2048 x 6144 11.7 / 12.4 / 11.5 ; 3072 x 9216 21.5 / 27.2 / 21.3 ; 4096 x 16384 38.3 / 40.4 / 30.7
//   units, 32 bits    1024 x 4096 7.3 / 7.5 ; 1536 x 6144 11.6 / 12.9 ; 2048 x 8192 18.0 / 17.0 ; 3072 x 9216 31.3 / 30.1 ; 4096 x 24576 83.9 / 87.8
template <bool BF16W, class Op>
static int pb_launch_matvec(cc_device* dev, const cc_buf* w, const Op& op, float* out, int64_t m, int64_t k, int64_t T, int accumulate) {
    const int64_t sms = dev->sm_count;
    // as many warps per row as there are too few rows for the device's warps, and, for the operand in registers, as the row's columns need for one block each
    auto split_for = [&](int warps, bool in_registers) {
        int split = 1;
        while (split < warps && (m * split * 2 <= sms * warps || (in_registers && k > (int64_t)split * PB_COLS))) split *= 2;
        return split;
    };
    const int half = split_for(16, true), full = split_for(32, true);
    bool registers;
    if (Op::NORM) registers = BF16W || k > PB_COLS / 2 || m <= 64 * sms;
    else registers = m >= 2048 || (BF16W && k > (int64_t)full * (PB_COLS * 3 / 4));
    if (!registers) return pb_launch_matvec_by<Op>(dev, pb_matvec_shared_kernel<BF16W, Op>, 1024, w, op, out, m, k, T, accumulate, split_for(32, false));
    auto by = [&](auto threads, int split) {
        return pb_launch_matvec_by<Op>(dev, pb_matvec_kernel<BF16W, Op, decltype(threads)::value>, decltype(threads)::value, w, op, out, m, k, T, accumulate, split);
    };
    if constexpr (BF16W && !Op::NORM) return by(std::integral_constant<int, 1024>{}, full);
    else {
        if constexpr (BF16W) { if (m * half > 8 * 16 * sms) return by(std::integral_constant<int, 1024>{}, full); }      // more than 8 turns of 16 warps
        return by(std::integral_constant<int, 512>{}, half);
    }
}
static bool pb_tensor_cores(const cc_buf* w, int64_t m, int64_t k, int64_t T) {
    return w->dtype == CC_BF16 && cc_prefill_bf16_supported(m, k, T) && ((uintptr_t)w->plane[0] & 15) == 0;
}

#define PB_ENTER(dev, what)                                                                                           \
    if (!(dev)) return CC_ERR_ARG;                                                                                    \
    CC_ENTER(dev);                                                                                                    \
    if (LAZY(dev)) return cc_fail((dev), CC_ERR_UNSUPPORTED, "%s: not available on a lazy (graph / megakernel) device", what)
#define PB_VIEW(dev, v, what)                                                                                         \
    do {                                                                                                              \
        if (!view_ok(v)) return cc_fail((dev), CC_ERR_ARG, "%s: bad tensor view", what);                              \
        if (!view_in_bounds(v)) return cc_fail((dev), CC_ERR_TENSOR, "%s: view addresses element %lld of a buffer of %lld", what, \
                                               (long long)view_max_offset(v), (long long)(v)->buf->nelems);           \
    } while (0)
#define PB_F32(dev, v, what)                                                        \
    do {                                                                            \
        PB_VIEW(dev, v, what);                                                      \
        REQUIRE_F32(dev, v, what);                                                  \
        CC_REQUIRE(dev, view_contiguous(v), "%s: not contiguous", what);            \
    } while (0)
#define PB_MATRIX(dev, v, what)                                                                                                                            \
    do {                                                                                                                                                   \
        PB_VIEW(dev, v, what);                                                                                                                             \
        CC_REQUIRE(dev, (v)->ndim == 2 && view_contiguous(v) && ((v)->buf->dtype == CC_F32 || (v)->buf->dtype == CC_BF16), "%s: an F32 or BF16 matrix is needed", what); \
    } while (0)
static inline const float* pb_ptr(const cc_view* v) { return (const float*)v->buf->plane[0]; }

extern "C" CC_API int cc_layer_norm_product(cc_device* dev, const cc_view* x, const cc_view* norm_w, const cc_view* norm_b, float eps, const cc_view* w, cc_buf** out) {
    PB_ENTER(dev, "layer_norm_product");
    if (!out) return cc_fail(dev, CC_ERR_ARG, "layer_norm_product: out is NULL");
    PB_F32(dev, x, "layer_norm_product x"); PB_F32(dev, norm_w, "layer_norm_product norm_w"); PB_MATRIX(dev, w, "layer_norm_product w");
    if (norm_b) PB_F32(dev, norm_b, "layer_norm_product norm_b");
    CC_REQUIRE(dev, x->ndim == 2 && x->shape[1] >= 1 && w->shape[1] == x->shape[1] && view_len(norm_w) == x->shape[1] && (!norm_b || view_len(norm_b) == x->shape[1]),
               "layer_norm_product: x must be [T, k], the norm's weight (and bias) [k] and w [m, k]");
    const int64_t T = x->shape[0], k = x->shape[1], m = w->shape[0];
    cc_buf* o = nullptr;
    int rc = cc_new_activation(dev, T * m, CC_F32, false, &o);
    if (rc) return rc;
    *out = o;
    if (T == 0 || m == 0) return CC_OK;
    const float *xp = pb_ptr(x), *nw = pb_ptr(norm_w), *nb = norm_b ? pb_ptr(norm_b) : nullptr;
    if (pb_few(T, k)) {
        const PbNorm op = {xp, nw, nb, eps};
        return w->buf->dtype == CC_BF16 ? pb_launch_matvec<true>(dev, w->buf, op, (float*)o->base, m, k, T, 0) : pb_launch_matvec<false>(dev, w->buf, op, (float*)o->base, m, k, T, 0);
    }
    if (pb_tensor_cores(w->buf, m, k, T)) {
        void* operand = nullptr;
        rc = cc_prefill_bf16_operand(dev, T, k, &operand);
        if (rc) return rc;
        cc_launch_pdl(dev, pb_norm_bf16_kernel, (unsigned)T, PB_LN_THREADS, 0, xp, nw, nb, (__nv_bfloat16*)operand, (int)k, eps);
        CC_LAUNCH_CHECK(dev);
        return cc_launch_prefill_bf16_operand(dev, w->buf, (float*)o->base, m, k, T, 0);
    }
    void* h = nullptr; size_t cls = 0;
    rc = cc_pool_alloc(dev, (size_t)T * k * 4, &h, &cls);
    if (rc) return rc;
    cc_launch_pdl(dev, pb_norm_f32_kernel, (unsigned)T, PB_LN_THREADS, 0, xp, nw, nb, (float*)h, (int)k, eps);
    dev->launches++;
    rc = cc_launch_dense_tile(dev, w->buf, (const float*)h, (float*)o->base, m, k, T, 0);
    cc_pool_free(dev, h, cls);
    return rc;
}

extern "C" CC_API int cc_joined_product_accumulate(cc_device* dev, const cc_view* dst, const cc_view* w, const cc_view* a, const cc_view* src, int32_t gate_col0, int32_t up_col0, int32_t ff,
                                                   const cc_glu_params* glu) {
    PB_ENTER(dev, "joined_product_accumulate");
    PB_F32(dev, dst, "joined_product_accumulate dst"); PB_MATRIX(dev, w, "joined_product_accumulate w"); PB_F32(dev, a, "joined_product_accumulate a");
    CC_REQUIRE(dev, dst->ndim == 2 && a->ndim == 2 && a->shape[0] == dst->shape[0] && ff >= 0 && w->shape[0] == dst->shape[1] && w->shape[1] == a->shape[1] + ff,
               "joined_product_accumulate: dst must be [T, m], a [T, ca] and w [m, ca + ff]");
    const int64_t T = dst->shape[0], m = dst->shape[1], k = w->shape[1];
    PbJoin op{};
    op.a = pb_ptr(a); op.ca = (int)a->shape[1]; op.ff = ff;
    if (ff > 0) {
        if (!src || !glu) return cc_fail(dev, CC_ERR_ARG, "joined_product_accumulate: the gated units need their numbers and constants");
        PB_VIEW(dev, src, "joined_product_accumulate src");
        REQUIRE_F32(dev, src, "joined_product_accumulate src");
        CC_REQUIRE(dev, src->ndim == 2 && src->strides[1] == 1 && src->strides[0] >= src->shape[1] && src->shape[0] == T && gate_col0 >= 0 && up_col0 >= 0 &&
                            (int64_t)gate_col0 + ff <= src->shape[1] && (int64_t)up_col0 + ff <= src->shape[1],
                   "joined_product_accumulate: src needs %d columns from columns %d and %d on", ff, gate_col0, up_col0);
        op.g = pb_ptr(src) + gate_col0; op.u = pb_ptr(src) + up_col0; op.rs = src->strides[0]; op.P = *glu;
    }
    if (T == 0 || m == 0) return CC_OK;
    float* out = (float*)dst->buf->plane[0];
    if (pb_few(T, k)) return w->buf->dtype == CC_BF16 ? pb_launch_matvec<true>(dev, w->buf, op, out, m, k, T, 1) : pb_launch_matvec<false>(dev, w->buf, op, out, m, k, T, 1);
    CC_REQUIRE(dev, T <= 65535, "joined_product_accumulate: %lld rows are too many for one pass", (long long)T);
    if (pb_tensor_cores(w->buf, m, k, T)) {
        void* operand = nullptr;
        int rc = cc_prefill_bf16_operand(dev, T, k, &operand);
        if (rc) return rc;
        const bool whole = op.ca % 8 == 0 && ff % 8 == 0 && op.rs % 4 == 0 && (((uintptr_t)op.a | (uintptr_t)op.g | (uintptr_t)op.u | (uintptr_t)operand) & 15) == 0;
        if (whole) cc_launch_pdl(dev, op.P.act == CC_ACT_SWISH ? pb_join8_bf16_kernel<true> : pb_join8_bf16_kernel<false>, dim3((unsigned)((k / 8 + 127) / 128), (unsigned)T), 128, 0, op, (__nv_bfloat16*)operand, (int)k);
        else cc_launch_pdl(dev, pb_join_bf16_kernel, dim3((unsigned)((k / 2 + 255) / 256), (unsigned)T), 256, 0, op, (__nv_bfloat16*)operand, (int)k);
        CC_LAUNCH_CHECK(dev);
        return cc_launch_prefill_bf16_operand(dev, w->buf, out, m, k, T, 1);
    }
    void* h = nullptr; size_t cls = 0;
    int rc = cc_pool_alloc(dev, (size_t)T * k * 4, &h, &cls);
    if (rc) return rc;
    cc_launch_pdl(dev, pb_join_f32_kernel, dim3((unsigned)((k + 255) / 256), (unsigned)T), 256, 0, op, (float*)h, (int)k);
    dev->launches++;
    rc = cc_launch_dense_tile(dev, w->buf, (const float*)h, out, m, k, T, 1);
    cc_pool_free(dev, h, cls);
    return rc;
}
