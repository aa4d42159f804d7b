// seqops.cu -- sequence-mixing and normalisation ops of include/crabml_seqops.h: norms on the sublayer output, the short causal
// convolution, the gated delta rule, and sliding-window attention over a ring cache.  Everything here is computed in 32-bit floats
// (explicit fmaf; expf / logf / log1pf of the CUDA math library, not the fast intrinsics); attention of many rows takes its two products on the tensor
// cores from 32-bit operands cut into bfloat16 numbers, with an error no larger than 32-bit sums have (split_gemm.cuh).
//
// One property every kernel keeps: the value computed for a token depends only on that token's inputs and on the state / cache
// contents, never on how many tokens the call carries or where the token sits in the call.  Sums run in a fixed order per output
// (a warp's lane-strided partial sums and the xor butterfly, one thread's sequential loop, or steps at fixed positions), so prefill, chunked prefill and
// token-by-token decoding give the same bits for the recurrent layers.  Attention has two ways, for calls of many rows and of few: a (query, key set) has the
// same bits in all calls that go one way, and differs between the two by the rounding of its sums.
#include <cooperative_groups.h>
#include <cuda.h>
#include <cuda_bf16.h>

#include "../../include/crabml_seqops.h"
#include "act.cuh"
#include "capi_checks.cuh"
#include "layer_norm.cuh"
#include "split_gemm.cuh"

#define SEQ_ENTER(dev, what)                                                                                          \
    if (!(dev)) return CC_ERR_ARG;                                                                                    \
    CC_ENTER(dev);                                                                                                    \
    if (LAZY(dev)) return cc_fail((dev), CC_ERR_UNSUPPORTED, "%s: not available on a lazy (graph / megakernel) device", what)
#define SEQ_VIEW(dev, v, what)                                                                                        \
    do {                                                                                                              \
        if (!view_ok(v)) return cc_fail((dev), CC_ERR_ARG, "%s: bad tensor view", what);                              \
        if (!view_in_bounds(v)) return cc_fail((dev), CC_ERR_TENSOR, "%s: view addresses element %lld of a buffer of %lld", what, \
                                               (long long)view_max_offset(v), (long long)(v)->buf->nelems);           \
        CC_REQUIRE(dev, view_contiguous(v), "%s: not contiguous", what);                                              \
    } while (0)
#define SEQ_F32(dev, v, what)                \
    do {                                     \
        SEQ_VIEW(dev, v, what);              \
        REQUIRE_F32(dev, v, what);           \
    } while (0)
// rows of a wider matrix (a column block, or the whole): unit column stride, any row stride that holds a row
#define SEQ_ROWS(dev, v, what)                                                                                        \
    do {                                                                                                              \
        if (!view_ok(v)) return cc_fail((dev), CC_ERR_ARG, "%s: bad tensor view", what);                              \
        if (!view_in_bounds(v)) return cc_fail((dev), CC_ERR_TENSOR, "%s: view addresses element %lld of a buffer of %lld", what, \
                                               (long long)view_max_offset(v), (long long)(v)->buf->nelems);           \
        REQUIRE_F32(dev, v, what);                                                                                    \
        CC_REQUIRE(dev, (v)->ndim == 2 && (v)->strides[1] == 1 && (v)->strides[0] >= (v)->shape[1], "%s: not rows of a matrix", what); \
    } while (0)
static inline float* fptr(const cc_view* v) { return (float*)v->buf->plane[0]; }

__device__ __forceinline__ float seq_sigmoid(float z) { return act_sigmoid(z); }
__device__ __forceinline__ float seq_softplus(float z) { return fmaxf(z, 0.0f) + log1pf(expf(-fabsf(z))); }
__device__ __forceinline__ float seq_act(float z, int act) { return act_apply(z, act); }

extern "C" CC_API int cc_tensor_zero(cc_device* dev, const cc_view* x) {
    SEQ_ENTER(dev, "tensor_zero");
    SEQ_VIEW(dev, x, "tensor_zero");
    const size_t esz = cc_block_bytes(x->buf->dtype);
    CC_REQUIRE(dev, !cc_is_quant(x->buf->dtype), "tensor_zero: plain types only");
    if (view_len(x)) CC_CUDA(dev, cudaMemsetAsync(x->buf->plane[0], 0, (size_t)view_len(x) * esz, dev->stream));
    return CC_OK;
}

// ---- norms --------------------------------------------------------------------------------------------------------------------
// one warp per row: lane-strided sum of squares, butterfly, then the scaled write
__global__ void rms_norm_gain_kernel(float* __restrict__ dst, const float* __restrict__ y, const float* __restrict__ gain, int gain_n, int rows, int cols,
                                     float eps, int accumulate, float mult) {
    pdl_enter();
    const int r = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (r >= rows) return;
    const float* yr = y + (int64_t)r * cols;
    float ss = 0.0f;
    for (int c = lane; c < cols; c += 32) ss = fmaf(yr[c], yr[c], ss);
    ss = warp_sum(ss);
    const float inv = 1.0f / sqrtf(ss / (float)cols + eps);
    float* dr = dst + (int64_t)r * cols;
    for (int c = lane; c < cols; c += 32) {
        const float v = yr[c] * inv * gain[gain_n == 1 ? 0 : c] * mult;
        dr[c] = accumulate ? dr[c] + v : v;
    }
}
// a wide row: one CTA per row, so that a call of few rows does not walk it with a single warp.  Thread-strided sums, the butterfly, then the
// warps' sums in warp order: the order depends on the row's length alone
#define RNG_THREADS 256
__global__ void __launch_bounds__(RNG_THREADS) rms_norm_gain_wide_kernel(float* __restrict__ dst, const float* __restrict__ y, const float* __restrict__ gain, int gain_n, int cols,
                                                                         float eps, int accumulate, float mult) {
    pdl_enter();
    __shared__ float red[RNG_THREADS / 32];
    const float* yr = y + (int64_t)blockIdx.x * cols;
    float* dr = dst + (int64_t)blockIdx.x * cols;
    float ss = 0.0f;
    for (int c = threadIdx.x; c < cols; c += RNG_THREADS) ss = fmaf(yr[c], yr[c], ss);
    ss = warp_sum(ss);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
    __syncthreads();
    float tot = 0.0f;
#pragma unroll
    for (int w = 0; w < RNG_THREADS / 32; w++) tot += red[w];
    const float inv = 1.0f / sqrtf(tot / (float)cols + eps);
    for (int c = threadIdx.x; c < cols; c += RNG_THREADS) {
        const float v = yr[c] * inv * gain[gain_n == 1 ? 0 : c] * mult;
        dr[c] = accumulate ? dr[c] + v : v;
    }
}
static int rms_norm_gain_impl(cc_device* dev, const cc_view* dst, const cc_view* y, const cc_view* gain, float eps, int32_t accumulate, float mult) {
    SEQ_ENTER(dev, "rms_norm_gain");
    SEQ_F32(dev, dst, "rms_norm_gain dst"); SEQ_F32(dev, y, "rms_norm_gain y"); SEQ_F32(dev, gain, "rms_norm_gain gain");
    CC_REQUIRE(dev, dst->ndim == 2 && y->ndim == 2 && dst->shape[0] == y->shape[0] && dst->shape[1] == y->shape[1], "rms_norm_gain: dst and y must be [rows, cols]");
    const int64_t rows = y->shape[0], cols = y->shape[1], gn = view_len(gain);
    CC_REQUIRE(dev, gn == 1 || gn == cols, "rms_norm_gain: gain has %lld elements, need 1 or %lld", (long long)gn, (long long)cols);
    if (rows == 0) return CC_OK;
    if (cols >= 512) cc_launch_pdl(dev, rms_norm_gain_wide_kernel, (unsigned)rows, RNG_THREADS, 0, fptr(dst), fptr(y), fptr(gain), (int)gn, (int)cols, eps, accumulate, mult);
    else cc_launch_pdl(dev, rms_norm_gain_kernel, (unsigned)((rows + 7) / 8), 256, 0, fptr(dst), fptr(y), fptr(gain), (int)gn, (int)rows, (int)cols, eps, accumulate, mult);
    CC_LAUNCH_CHECK(dev);
    return CC_OK;
}
extern "C" CC_API int cc_rms_norm_gain(cc_device* dev, const cc_view* dst, const cc_view* y, const cc_view* gain, float eps, int32_t accumulate) {
    return rms_norm_gain_impl(dev, dst, y, gain, eps, accumulate, 1.0f);
}
extern "C" CC_API int cc_rms_norm_gain_mult(cc_device* dev, const cc_view* dst, const cc_view* y, const cc_view* gain, float eps, float mult) {
    return rms_norm_gain_impl(dev, dst, y, gain, eps, 1, mult);
}

// one warp per (row, head)
// w_heads: how many heads have weights of their own (1: one vector for all)
__global__ void gated_head_rms_norm_kernel(float* __restrict__ x, const float* __restrict__ gate, const float* __restrict__ w, int64_t n_units, int hs, float eps, int act,
                                           int w_heads) {
    pdl_enter();
    const int64_t u = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (u >= n_units) return;
    float* xr = x + u * hs;
    const float* gr = gate ? gate + u * hs : nullptr;
    const float* wr = w ? w + (u % w_heads) * hs : nullptr;
    float ss = 0.0f;
    for (int c = lane; c < hs; c += 32) ss = fmaf(xr[c], xr[c], ss);
    ss = warp_sum(ss);
    const float inv = 1.0f / sqrtf(ss / (float)hs + eps);
    for (int c = lane; c < hs; c += 32) {
        float v = xr[c] * inv;
        if (wr) v *= wr[c];
        if (gr) v *= seq_act(gr[c], act);
        xr[c] = v;
    }
}
extern "C" CC_API int cc_gated_head_rms_norm(cc_device* dev, const cc_view* x, const cc_view* gate, const cc_view* w, int32_t head_size, float eps, int32_t gate_act) {
    SEQ_ENTER(dev, "gated_head_rms_norm");
    SEQ_F32(dev, x, "gated_head_rms_norm x");
    if (gate) SEQ_F32(dev, gate, "gated_head_rms_norm gate");
    if (w) SEQ_F32(dev, w, "gated_head_rms_norm w");
    const int64_t n = view_len(x);
    CC_REQUIRE(dev, head_size > 0 && n % head_size == 0 && (!gate || view_len(gate) == n), "gated_head_rms_norm: shapes do not fit head_size %d", head_size);
    int w_heads = 1;
    if (w && view_len(w) != head_size) {
        CC_REQUIRE(dev, x->ndim == 2 && view_len(w) == x->shape[1], "gated_head_rms_norm: w must have head_size elements or one per column");
        w_heads = (int)(x->shape[1] / head_size);
    }
    const int64_t units = n / head_size;
    if (!units) return CC_OK;
    cc_launch_pdl(dev, gated_head_rms_norm_kernel, (unsigned)((units + 7) / 8), 256, 0, fptr(x), gate ? fptr(gate) : nullptr, w ? fptr(w) : nullptr, units, head_size, eps, gate_act,
                                                                                    w_heads);
    CC_LAUNCH_CHECK(dev);
    return CC_OK;
}

__global__ void glu_kernel(float* __restrict__ g, const float* __restrict__ u, int64_t n, int act) {
    pdl_enter();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) g[i] = seq_act(g[i], act) * u[i];
}
extern "C" CC_API int cc_glu_inplace(cc_device* dev, const cc_view* gate, const cc_view* up, int32_t act) {
    SEQ_ENTER(dev, "glu_inplace");
    SEQ_F32(dev, gate, "glu_inplace gate"); SEQ_F32(dev, up, "glu_inplace up");
    const int64_t n = view_len(gate);
    CC_REQUIRE(dev, view_len(up) == n, "glu_inplace: sizes differ");
    if (!n) return CC_OK;
    cc_launch_pdl(dev, glu_kernel, (unsigned)((n + 255) / 256), 256, 0, fptr(gate), fptr(up), n, act);
    CC_LAUNCH_CHECK(dev);
    return CC_OK;
}
__global__ void activate_kernel(float* __restrict__ x, int64_t n, int act) {
    pdl_enter();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) x[i] = seq_act(x[i], act);
}
extern "C" CC_API int cc_activate_inplace(cc_device* dev, const cc_view* x, int32_t act) {
    SEQ_ENTER(dev, "activate_inplace");
    SEQ_F32(dev, x, "activate_inplace x");
    const int64_t n = view_len(x);
    if (!n) return CC_OK;
    cc_launch_pdl(dev, activate_kernel, (unsigned)((n + 255) / 256), 256, 0, fptr(x), n, act);
    CC_LAUNCH_CHECK(dev);
    return CC_OK;
}
__global__ void softcap_kernel(float* __restrict__ x, int64_t n, float cap) {
    pdl_enter();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) x[i] = cap * tanhf(x[i] / cap);
}
extern "C" CC_API int cc_softcap_inplace(cc_device* dev, const cc_view* x, float cap) {
    SEQ_ENTER(dev, "softcap_inplace");
    SEQ_F32(dev, x, "softcap_inplace x");
    CC_REQUIRE(dev, cap > 0.0f, "softcap_inplace: the cap must be positive");
    const int64_t n = view_len(x);
    if (!n) return CC_OK;
    cc_launch_pdl(dev, softcap_kernel, (unsigned)((n + 255) / 256), 256, 0, fptr(x), n, cap);
    CC_LAUNCH_CHECK(dev);
    return CC_OK;
}
// gate | up side by side in one product's rows
__global__ void glu_halves_kernel(const float* __restrict__ src, const float* __restrict__ bias, float* __restrict__ out, int64_t n, int ff, int act) {
    pdl_enter();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int64_t r = i / ff;
    const int c = (int)(i - r * ff);
    float g = src[r * 2 * ff + c], u = src[r * 2 * ff + ff + c];
    if (bias) { g += bias[c]; u += bias[ff + c]; }
    out[i] = seq_act(g, act) * u;
}
extern "C" CC_API int cc_glu_halves(cc_device* dev, const cc_view* src, const cc_view* bias, int32_t act, cc_buf** out) {
    SEQ_ENTER(dev, "glu_halves");
    if (!out) return cc_fail(dev, CC_ERR_ARG, "glu_halves: out is NULL");
    SEQ_F32(dev, src, "glu_halves src");
    CC_REQUIRE(dev, src->ndim == 2 && src->shape[1] % 2 == 0, "glu_halves: src must be [rows, 2 * ff]");
    const int64_t rows = src->shape[0], ff = src->shape[1] / 2;
    if (bias) { SEQ_F32(dev, bias, "glu_halves bias"); CC_REQUIRE(dev, view_len(bias) == 2 * ff, "glu_halves: the bias needs one number per column of src"); }
    cc_buf* o = nullptr;
    int rc = cc_new_activation(dev, rows * ff, CC_F32, false, &o);
    if (rc) return rc;
    *out = o;
    const int64_t n = rows * ff;
    if (!n) return CC_OK;
    cc_launch_pdl(dev, glu_halves_kernel, (unsigned)((n + 255) / 256), 256, 0, fptr(src), bias ? fptr(bias) : nullptr, (float*)o->base, n, (int)ff, act);
    CC_LAUNCH_CHECK(dev);
    return CC_OK;
}
__global__ void add_row_bias_kernel(float* __restrict__ x, const float* __restrict__ b, int64_t n, int cols) {
    pdl_enter();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) x[i] += b[i % cols];
}
extern "C" CC_API int cc_add_row_bias(cc_device* dev, const cc_view* x, const cc_view* bias) {
    SEQ_ENTER(dev, "add_row_bias");
    SEQ_F32(dev, x, "add_row_bias x"); SEQ_F32(dev, bias, "add_row_bias bias");
    CC_REQUIRE(dev, x->ndim == 2 && view_len(bias) == x->shape[1], "add_row_bias: x must be [rows, cols] and bias [cols]");
    const int64_t n = view_len(x);
    if (!n) return CC_OK;
    cc_launch_pdl(dev, add_row_bias_kernel, (unsigned)((n + 255) / 256), 256, 0, fptr(x), fptr(bias), n, (int)x->shape[1]);
    CC_LAUNCH_CHECK(dev);
    return CC_OK;
}
__global__ void scaled_sum_kernel(float* __restrict__ dst, const float* __restrict__ a, float sa, const float* __restrict__ b, float sb, int64_t n) {
    pdl_enter();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[i] = sa * a[i] + sb * b[i];
}
extern "C" CC_API int cc_scaled_sum(cc_device* dev, const cc_view* dst, const cc_view* a, float sa, const cc_view* b, float sb) {
    SEQ_ENTER(dev, "scaled_sum");
    SEQ_F32(dev, dst, "scaled_sum dst"); SEQ_F32(dev, a, "scaled_sum a"); SEQ_F32(dev, b, "scaled_sum b");
    const int64_t n = view_len(dst);
    CC_REQUIRE(dev, view_len(a) == n && view_len(b) == n, "scaled_sum: sizes differ");
    if (!n) return CC_OK;
    cc_launch_pdl(dev, scaled_sum_kernel, (unsigned)((n + 255) / 256), 256, 0, fptr(dst), fptr(a), sa, fptr(b), sb, n);
    CC_LAUNCH_CHECK(dev);
    return CC_OK;
}

__global__ void scaled_sum_accumulate_kernel(float* __restrict__ dst, const float* __restrict__ a, float sa, const float* __restrict__ b, float sb, const float* __restrict__ c,
                                             int64_t n) {
    pdl_enter();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float v = sa * a[i] + sb * b[i];
    if (c) v += c[i];
    dst[i] += v;
}
extern "C" CC_API int cc_scaled_sum_accumulate(cc_device* dev, const cc_view* dst, const cc_view* a, float sa, const cc_view* b, float sb, const cc_view* c) {
    SEQ_ENTER(dev, "scaled_sum_accumulate");
    SEQ_F32(dev, dst, "scaled_sum_accumulate dst"); SEQ_F32(dev, a, "scaled_sum_accumulate a"); SEQ_F32(dev, b, "scaled_sum_accumulate b");
    if (c) SEQ_F32(dev, c, "scaled_sum_accumulate c");
    const int64_t n = view_len(dst);
    CC_REQUIRE(dev, view_len(a) == n && view_len(b) == n && (!c || view_len(c) == n), "scaled_sum_accumulate: sizes differ");
    if (!n) return CC_OK;
    cc_launch_pdl(dev, scaled_sum_accumulate_kernel, (unsigned)((n + 255) / 256), 256, 0, fptr(dst), fptr(a), sa, fptr(b), sb, c ? fptr(c) : nullptr, n);
    CC_LAUNCH_CHECK(dev);
    return CC_OK;
}
// one gate number per (row, head): one thread per element
__global__ void head_gate_kernel(float* __restrict__ x, const float* __restrict__ g, int64_t n, int hs, int heads, int64_t grs, int act) {
    pdl_enter();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int64_t u = i / hs, t = u / heads;
    x[i] *= seq_act(g[t * grs + (u - t * heads)], act);
}
// the same, four neighbouring elements of a head per thread: grid (columns / 512, rows).  512 x 8 heads of 128, us: one element by 64-bit divisions 5.0 ; here 4.0
__global__ void __launch_bounds__(128) head_gate4_kernel(float* __restrict__ x, const float* __restrict__ g, int cols, int hs, int64_t grs, int act) {
    pdl_enter();
    const int c = (blockIdx.x * 128 + threadIdx.x) * 4;
    if (c >= cols) return;
    float4* at = (float4*)(x + (int64_t)blockIdx.y * cols + c);
    float4 v = *at;
    const float f = seq_act(g[blockIdx.y * grs + c / hs], act);
    v.x *= f; v.y *= f; v.z *= f; v.w *= f;
    *at = v;
}
// gate numbers in the columns col0 .. col0 + n_heads of g's rows
static int head_gate_impl(cc_device* dev, const cc_view* x, const cc_view* g, int32_t col0, int32_t n_heads, int32_t act) {
    SEQ_F32(dev, x, "head_gate x"); SEQ_ROWS(dev, g, "head_gate g");
    CC_REQUIRE(dev, x->ndim == 2 && n_heads > 0 && x->shape[1] % n_heads == 0 && g->shape[0] == x->shape[0] && col0 >= 0 && (int64_t)col0 + n_heads <= g->shape[1],
               "head_gate: x must be [rows, heads * head_size] and g hold %d columns from column %d on", n_heads, col0);
    const int64_t n = view_len(x);
    if (!n) return CC_OK;
    const int64_t hs = x->shape[1] / n_heads, cols = x->shape[1];
    if (hs % 4 == 0 && x->shape[0] <= 65535 && ((uintptr_t)fptr(x) & 15) == 0)
        cc_launch_pdl(dev, head_gate4_kernel, dim3((unsigned)((cols / 4 + 127) / 128), (unsigned)x->shape[0]), 128, 0, fptr(x), fptr(g) + col0, (int)cols, (int)hs, g->strides[0], act);
    else cc_launch_pdl(dev, head_gate_kernel, (unsigned)((n + 255) / 256), 256, 0, fptr(x), fptr(g) + col0, n, (int)hs, n_heads, g->strides[0], act);
    CC_LAUNCH_CHECK(dev);
    return CC_OK;
}
extern "C" CC_API int cc_head_gate(cc_device* dev, const cc_view* x, const cc_view* g, int32_t n_heads, int32_t act) {
    SEQ_ENTER(dev, "head_gate");
    return head_gate_impl(dev, x, g, 0, n_heads, act);
}
extern "C" CC_API int cc_head_gate_cols(cc_device* dev, const cc_view* x, const cc_view* gate_src, int32_t gate_col0, int32_t n_heads, int32_t act) {
    SEQ_ENTER(dev, "head_gate");
    return head_gate_impl(dev, x, gate_src, gate_col0, n_heads, act);
}
// out = [a | b] row by row: one thread per element of out
__global__ void concat_cols_kernel(const float* __restrict__ a, const float* __restrict__ b, float* __restrict__ out, int64_t n, int ca, int cb) {
    pdl_enter();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int64_t r = i / (ca + cb);
    const int c = (int)(i - r * (ca + cb));
    out[i] = c < ca ? a[r * ca + c] : b[r * cb + (c - ca)];
}
extern "C" CC_API int cc_concat_cols(cc_device* dev, const cc_view* a, const cc_view* b, cc_buf** out) {
    SEQ_ENTER(dev, "concat_cols");
    if (!out) return cc_fail(dev, CC_ERR_ARG, "concat_cols: out is NULL");
    SEQ_F32(dev, a, "concat_cols a"); SEQ_F32(dev, b, "concat_cols b");
    CC_REQUIRE(dev, a->ndim == 2 && b->ndim == 2 && a->shape[0] == b->shape[0], "concat_cols: a and b must be [rows, ca] and [rows, cb]");
    const int64_t rows = a->shape[0], ca = a->shape[1], cb = b->shape[1];
    cc_buf* o = nullptr;
    int rc = cc_new_activation(dev, rows * (ca + cb), CC_F32, false, &o);
    if (rc) return rc;
    *out = o;
    const int64_t n = rows * (ca + cb);
    if (!n) return CC_OK;
    cc_launch_pdl(dev, concat_cols_kernel, (unsigned)((n + 255) / 256), 256, 0, fptr(a), fptr(b), (float*)o->base, n, (int)ca, (int)cb);
    CC_LAUNCH_CHECK(dev);
    return CC_OK;
}

// ---- a second embedding row chosen by a hash of the token pair ------------------------------------------------------------------------
// one thread per (token, column); the hash is taken in 64-bit integers
__global__ void pair_hash_rows_add_kernel(float* __restrict__ dst, const float* __restrict__ table, const int64_t* __restrict__ tok, const int32_t* __restrict__ last, int64_t n,
                                          int cols, int64_t mul_prev, int64_t mul_cur, int64_t buckets) {
    pdl_enter();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int64_t t = i / cols;
    const int c = (int)(i - t * cols);
    const int64_t prev = t > 0 ? tok[t - 1] : (int64_t)last[0] - 1;
    const int64_t row = prev < 0 ? buckets : (prev * mul_prev + tok[t] * mul_cur) % buckets;
    dst[i] += table[row * cols + c];
}
__global__ void pair_hash_last_kernel(const int64_t* __restrict__ tok, int32_t* __restrict__ last, int n) { pdl_enter(); last[0] = (int32_t)tok[n - 1] + 1; }
extern "C" CC_API int cc_pair_hash_rows_add(cc_device* dev, const cc_view* dst, const cc_view* table, const int64_t* tokens, int32_t n, int32_t slot, const cc_view* last,
                                            int64_t mul_prev, int64_t mul_cur, int64_t buckets) {
    SEQ_ENTER(dev, "pair_hash_rows_add");
    SEQ_F32(dev, dst, "pair_hash_rows_add dst"); SEQ_F32(dev, table, "pair_hash_rows_add table");
    SEQ_VIEW(dev, last, "pair_hash_rows_add last");
    CC_REQUIRE(dev, last->buf->dtype == CC_I32 && view_len(last) == 1, "pair_hash_rows_add: last must be I32 [1]");
    CC_REQUIRE(dev, dst->ndim == 2 && table->ndim == 2 && dst->shape[1] == table->shape[1] && buckets >= 1 && table->shape[0] == buckets + 1 && mul_prev >= 0 && mul_cur >= 0,
               "pair_hash_rows_add: dst must be [n, cols] and table [buckets + 1, cols]");
    CC_REQUIRE(dev, n >= 0 && dst->shape[0] == n && (tokens || (n == 1 && slot >= 0 && slot < CC_N_SLOTS)), "pair_hash_rows_add: %d tokens for %lld rows", n, (long long)dst->shape[0]);
    if (n == 0) return CC_OK;
    const int64_t* tok = nullptr;
    if (tokens) {
        for (int i = 0; i < n; i++) CC_REQUIRE(dev, tokens[i] >= 0 && tokens[i] < ((int64_t)1 << 31) - 1, "pair_hash_rows_add: token id %lld", (long long)tokens[i]);
        int rc = cc_ensure_dev_idx(dev, (size_t)n * 8);
        if (rc) return rc;
        CC_CUDA(dev, cudaMemcpyAsync(dev->dev_idx, tokens, (size_t)n * 8, cudaMemcpyHostToDevice, dev->stream));
        tok = (const int64_t*)dev->dev_idx;
    } else {
        int rc = cc_ensure_slots(dev);
        if (rc) return rc;
        tok = dev->slots + slot;
    }
    const int64_t total = (int64_t)n * dst->shape[1];
    int32_t* lp = (int32_t*)last->buf->plane[0];
    cc_launch_pdl(dev, pair_hash_rows_add_kernel, (unsigned)((total + 255) / 256), 256, 0, fptr(dst), fptr(table), tok, lp, total, (int)dst->shape[1], mul_prev, mul_cur, buckets);
    dev->launches++;
    cc_launch_pdl(dev, pair_hash_last_kernel, 1, 1, 0, tok, lp, n);
    CC_LAUNCH_CHECK(dev);
    return CC_OK;
}

// ---- short causal convolution ----------------------------------------------------------------------------------------------------
// one warp per (token, run of hs channels).  in[t'] for t' < 0 comes from the tail: tail row (K-1) + t'.
// in_bias (or NULL) is added to every input of x as it is read; the tail holds inputs that already carry it (or the zeros before a sequence)
__global__ void short_conv_kernel(const float* __restrict__ x, const float* __restrict__ w, const float* __restrict__ bias, const float* __restrict__ tail,
                                  float* __restrict__ y, int T, int C, int K, int hs, int act, int unit, float ueps, float uscale, const float* __restrict__ in_bias, int64_t xrs) {
    pdl_enter();
    const int heads = C / hs;
    const int64_t u = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (u >= (int64_t)T * heads) return;
    const int t = (int)(u / heads), h = (int)(u % heads);
    float ss = 0.0f;
    for (int cc = lane; cc < hs; cc += 32) {
        const int c = h * hs + cc;
        float acc = bias ? bias[c] : 0.0f;
        for (int j = 0; j < K; j++) {
            const int ti = t - (K - 1) + j;
            const float v = ti >= 0 ? (in_bias ? x[ti * xrs + c] + in_bias[c] : x[ti * xrs + c]) : tail[(int64_t)(ti + K - 1) * C + c];
            acc = fmaf(w[(int64_t)c * K + j], v, acc);
        }
        acc = seq_act(acc, act);
        y[(int64_t)t * C + c] = acc;
        ss = fmaf(acc, acc, ss);
    }
    if (unit) {
        ss = warp_sum(ss);
        const float f = uscale / sqrtf(ss + ueps);
        for (int cc = lane; cc < hs; cc += 32) y[(int64_t)t * C + h * hs + cc] *= f;
    }
}
// tail <- the last K-1 rows of (tail ++ x); one thread per channel, ascending rows: row j is written after row T + j > j was read
__device__ __forceinline__ void short_conv_new_tail(const float* x, float* tail, int T, int C, int K, const float* in_bias, int64_t xrs, int c) {
    for (int j = 0; j < K - 1; j++) {
        const int ti = T + j - (K - 1);
        tail[(int64_t)j * C + c] = ti >= 0 ? (in_bias ? x[ti * xrs + c] + in_bias[c] : x[ti * xrs + c]) : tail[(int64_t)(ti + K - 1) * C + c];
    }
}
__global__ void short_conv_tail_kernel(const float* __restrict__ x, float* tail, int T, int C, int K, const float* __restrict__ in_bias, int64_t xrs) {
    pdl_enter();
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c < C) short_conv_new_tail(x, tail, T, C, K, in_bias, xrs, c);
}
// few rows (decoding): one thread per channel walks the rows and then renews its channel's tail -- one launch; the sums are those of
// short_conv_kernel
#define SC_FEW_ROWS 8
__global__ void short_conv_few_kernel(const float* __restrict__ x, const float* __restrict__ w, const float* __restrict__ bias, float* tail, float* __restrict__ y, int T, int C,
                                      int K, int act, const float* __restrict__ in_bias, int64_t xrs) {
    pdl_enter();
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= C) return;
    for (int t = 0; t < T; t++) {
        float acc = bias ? bias[c] : 0.0f;
        for (int j = 0; j < K; j++) {
            const int ti = t - (K - 1) + j;
            const float v = ti >= 0 ? (in_bias ? x[ti * xrs + c] + in_bias[c] : x[ti * xrs + c]) : tail[(int64_t)(ti + K - 1) * C + c];
            acc = fmaf(w[(int64_t)c * K + j], v, acc);
        }
        y[(int64_t)t * C + c] = seq_act(acc, act);
    }
    short_conv_new_tail(x, tail, T, C, K, in_bias, xrs, c);
}
static int short_conv_impl(cc_device* dev, const cc_view* x, const cc_view* w, const cc_view* bias, const cc_view* tail, int32_t act, int32_t head_size, int32_t unit_norm,
                           float unit_eps, float unit_scale, cc_buf** out, const cc_view* in_bias = nullptr, int64_t col0 = -1) {
    SEQ_ENTER(dev, "short_conv");
    if (!out) return cc_fail(dev, CC_ERR_ARG, "short_conv: out is NULL");
    SEQ_F32(dev, x, "short_conv x"); SEQ_F32(dev, w, "short_conv w");
    CC_REQUIRE(dev, x->ndim == 2 && w->ndim == 2 && (col0 < 0 ? w->shape[0] == x->shape[1] : col0 + w->shape[0] <= x->shape[1]),
               "short_conv: x must be [T, C] (or hold C columns from column %lld on) and w [C, K]", (long long)col0);
    const int64_t T = x->shape[0], C = w->shape[0], K = w->shape[1], xrs = x->shape[1];
    const float* xp = fptr(x) + (col0 < 0 ? 0 : col0);
    CC_REQUIRE(dev, K >= 1, "short_conv: no taps");
    if (K > 1) {
        SEQ_F32(dev, tail, "short_conv tail");
        CC_REQUIRE(dev, view_len(tail) == (K - 1) * C, "short_conv: tail must be [K-1, C]");
    }
    int hs = head_size > 0 ? head_size : (int)C;
    CC_REQUIRE(dev, C % hs == 0, "short_conv: head_size %d does not divide %lld channels", hs, (long long)C);
    if (!unit_norm) {            // nothing ties the channels of a head together: a warp takes the widest run of at most 32 channels that divides C
        hs = 32;
        while (C % hs) hs--;
    }
    if (bias) { SEQ_F32(dev, bias, "short_conv bias"); CC_REQUIRE(dev, view_len(bias) == C, "short_conv: the bias needs one number per channel"); }
    if (in_bias) { SEQ_F32(dev, in_bias, "short_conv in_bias"); CC_REQUIRE(dev, view_len(in_bias) == C, "short_conv: the input bias needs one number per channel"); }
    const float* ibp = in_bias ? fptr(in_bias) : nullptr;
    cc_buf* y = nullptr;
    int rc = cc_new_activation(dev, T * C, CC_F32, false, &y);
    if (rc) return rc;
    *out = y;
    if (T == 0) return CC_OK;
    const float* tp = K > 1 ? fptr(tail) : nullptr;
    if (K > 1 && T <= SC_FEW_ROWS && !unit_norm) {
        cc_launch_pdl(dev, short_conv_few_kernel, (unsigned)((C + 127) / 128), 128, 0, xp, fptr(w), bias ? fptr(bias) : nullptr, fptr(tail), (float*)y->base, (int)T, (int)C, (int)K, act, ibp, xrs);
        CC_LAUNCH_CHECK(dev);
        return CC_OK;
    }
    const int64_t units = T * (C / hs);
    cc_launch_pdl(dev, short_conv_kernel, (unsigned)((units + 7) / 8), 256, 0, xp, fptr(w), bias ? fptr(bias) : nullptr, tp, (float*)y->base, (int)T, (int)C, (int)K, hs, act, unit_norm,
                                                                        unit_eps, unit_scale, ibp, xrs);
    CC_LAUNCH_CHECK(dev);
    if (K > 1) {
        cc_launch_pdl(dev, short_conv_tail_kernel, (unsigned)((C + 127) / 128), 128, 0, xp, fptr(tail), (int)T, (int)C, (int)K, ibp, xrs);
        CC_LAUNCH_CHECK(dev);
    }
    return CC_OK;
}

extern "C" CC_API int cc_short_conv(cc_device* dev, const cc_view* x, const cc_view* w, const cc_view* tail, int32_t act, int32_t head_size, int32_t unit_norm,
                                    float unit_eps, float unit_scale, cc_buf** out) {
    return short_conv_impl(dev, x, w, nullptr, tail, act, head_size, unit_norm, unit_eps, unit_scale, out);
}
extern "C" CC_API int cc_short_conv_biases(cc_device* dev, const cc_view* x, const cc_view* w, const cc_view* in_bias, const cc_view* bias, const cc_view* tail, int32_t act,
                                           cc_buf** out) {
    return short_conv_impl(dev, x, w, bias, tail, act, 0, 0, 0.0f, 1.0f, out, in_bias);
}
extern "C" CC_API int cc_short_conv_bias(cc_device* dev, const cc_view* x, const cc_view* w, const cc_view* bias, const cc_view* tail, int32_t act, cc_buf** out) {
    return short_conv_impl(dev, x, w, bias, tail, act, 0, 0, 0.0f, 1.0f, out);
}

extern "C" CC_API int cc_short_conv_cols(cc_device* dev, const cc_view* src, int32_t col0, const cc_view* w, const cc_view* bias, const cc_view* tail, int32_t act, cc_buf** out) {
    if (dev && col0 < 0) return cc_fail(dev, CC_ERR_ARG, "short_conv_cols: column %d", col0);
    return short_conv_impl(dev, src, w, bias, tail, act, 0, 0, 0.0f, 1.0f, out, nullptr, col0);
}

// ---- gated delta rule -------------------------------------------------------------------------------------------------------------
// beta / decay of every (token, head): bd[(t * H + h) * 2] = {sigmoid(b), exp(-exp(a_log) * softplus(a + dt_bias))}
__global__ void delta_gates_kernel(const float* __restrict__ a, const float* __restrict__ b, const float* __restrict__ a_log, const float* __restrict__ dt_bias,
                                   float* __restrict__ bd, int64_t n, int H) {
    pdl_enter();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int h = (int)(i % H);
    bd[i * 2] = seq_sigmoid(b[i]);
    bd[i * 2 + 1] = expf(-expf(a_log[h]) * seq_softplus(a[i] + dt_bias[h]));
}
// grid (H, ceil(dv / columns per CTA)).  A column j of the head's state S[dk][dv] is owned for the whole call by SPLIT adjacent threads,
// each holding dk / SPLIT of its entries: DK > 0 keeps them in registers (16 per thread: groups of 4, dealt in turn, so that a warp's reads of k and q
// fall into different banks), DK == 0 (any dk) in shared memory [dk][DR_THREADS].
// Tokens run in order; per token two passes over dk:
//   acc = sum_i S[i] k[i]           (the decayed read-out is decay * acc)
//   u = beta * (v - decay * acc) ;  S[i] = decay * S[i] + k[i] * u ;  out = sum_i S[i] q[i]
// k, q, v, beta and decay of DR_TB tokens at a time are staged in shared memory (one trip to L2 per block of tokens instead of several per
// token).  Both dot products run as four interleaved partial sums per thread (i mod 4), added as (p0 + p1) + (p2 + p3); the SPLIT shares of acc are
// added by a butterfly, those of out in ascending order after the block of tokens: a fixed order, the same for any T.
// Bound by the chain acc -> u -> S from token to token, which is why a column is cut into 16 entries per thread: with two threads per column of 128
// (64 CTAs of 2 warps for 16 heads) a token took 860 cycles, most of them issue slots of one warp.  1000 tokens, 16 heads (4 key heads) of 128:
// 439 -> 217 us.
#define DR_THREADS 64                                   // DK == 0
#define DR_SPLIT_THREADS 128                            // DK > 0
#define DR_TB 16
__device__ __forceinline__ void dr_cp_async16(float* dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void dr_cp_async4(float* dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
// one staging buffer: k[DR_TB][dk4], q[DR_TB][dk4], bd[DR_TB][2], v[DR_TB][columns]
__host__ __device__ constexpr int dr_stage_floats(int dk4, int cols) { return 2 * DR_TB * dk4 + 2 * DR_TB + DR_TB * cols; }
template <int DK, int SPLIT, int THREADS>
__global__ void __launch_bounds__(THREADS) delta_rule_kernel(const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ v,
                                                             const float* __restrict__ bd, float* __restrict__ state, float* __restrict__ o, int T, int H, int G,
                                                             int dk, int dv) {
    pdl_enter();
    extern __shared__ __align__(16) float dr_sm[];            // two staging buffers, then the state columns (DK == 0) or the shares of out (DK > 0)
    constexpr int DKP = DK > 0 ? DK / SPLIT : 4;
    constexpr int COLS = THREADS / SPLIT;
    const int dk4 = (dk + 3) & ~3;
    const int stage_floats = dr_stage_floats(dk4, COLS);
    const int h = blockIdx.x, g = h / (H / G);
    const int part = threadIdx.x % SPLIT, col = threadIdx.x / SPLIT;
    const int j0 = blockIdx.y * COLS, j = j0 + col;
    const bool live = j < dv;
    const int jj = live ? j : dv - 1;                       // idle threads shadow the last column and never store
    float S[DKP];
    float* rest = dr_sm + 2 * stage_floats;
    float* Ss = rest + threadIdx.x;                          // generic: S[i] at Ss[i * THREADS]
    float* sp = state + ((int64_t)h * dk + part * 4) * dv + jj;
    constexpr int TURN = 4 * SPLIT;                          // thread `part` holds the entries 4 part .. 4 part + 3 of every TURN
    if (DK > 0) {
#pragma unroll
        for (int i = 0; i < DKP; i++) S[i] = sp[(int64_t)((i >> 2) * TURN + (i & 3)) * dv];
    } else {
        for (int i = 0; i < dk4; i++) Ss[i * THREADS] = i < dk ? sp[(int64_t)i * dv] : 0.0f;
    }
    // the pad lanes dk .. dk4 of both buffers are zero for the whole call (the copies below never touch them)
    if (dk4 != dk)
        for (int idx = threadIdx.x; idx < 2 * 2 * DR_TB; idx += THREADS)
            for (int i = dk; i < dk4; i++) dr_sm[(idx / (2 * DR_TB)) * stage_floats + (idx % (2 * DR_TB)) * dk4 + i] = 0.0f;
    // asynchronous copies (cp.async) of a block of tokens: issued one block ahead, so the trip to L2 overlaps the recurrence
    auto stage = [&](int buf, int tb) {
        float* base = dr_sm + buf * stage_floats;
        const int nt = min(DR_TB, T - tb);
        if ((dk & 3) == 0) {
            const int per = dk >> 2;
            for (int idx = threadIdx.x; idx < nt * per; idx += THREADS) {
                const int tt = idx / per, c = (idx - tt * per) * 4;
                const int64_t src = ((int64_t)(tb + tt) * G + g) * dk + c;
                dr_cp_async16(base + tt * dk4 + c, k + src);
                dr_cp_async16(base + (DR_TB + tt) * dk4 + c, q + src);
            }
        } else {
            for (int idx = threadIdx.x; idx < nt * dk; idx += THREADS) {
                const int tt = idx / dk, c = idx - tt * dk;
                const int64_t src = ((int64_t)(tb + tt) * G + g) * dk + c;
                dr_cp_async4(base + tt * dk4 + c, k + src);
                dr_cp_async4(base + (DR_TB + tt) * dk4 + c, q + src);
            }
        }
        float* sbd = base + 2 * DR_TB * dk4;
        for (int idx = threadIdx.x; idx < nt * 2; idx += THREADS) dr_cp_async4(sbd + idx, bd + ((int64_t)(tb + (idx >> 1)) * H + h) * 2 + (idx & 1));
        float* sv = sbd + 2 * DR_TB;
        for (int idx = threadIdx.x; idx < nt * COLS; idx += THREADS) {
            const int tt = idx / COLS, c = idx - tt * COLS;
            dr_cp_async4(sv + idx, v + ((int64_t)(tb + tt) * H + h) * dv + min(j0 + c, dv - 1));
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (T > 0) stage(0, 0);
    int buf = 0;
    for (int tb = 0; tb < T; tb += DR_TB, buf ^= 1) {
        const int nt = min(DR_TB, T - tb);
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();                                      // this block has landed for everyone, and everyone is done with the other buffer
        if (tb + DR_TB < T) stage(buf ^ 1, tb + DR_TB);
        const float* base = dr_sm + buf * stage_floats;
        const float* sbd = base + 2 * DR_TB * dk4;
        const float* sv = sbd + 2 * DR_TB + col;
        const float* kt = base + part * 4;
        const float* qt = base + DR_TB * dk4 + part * 4;
#pragma unroll 1
        for (int tt = 0; tt < nt; tt++, kt += dk4, qt += dk4) {
            const float beta = sbd[tt * 2], dec = sbd[tt * 2 + 1];
            const float vj = sv[tt * COLS];
            float a0 = 0.0f, a1 = 0.0f, a2 = 0.0f, a3 = 0.0f, o0 = 0.0f, o1 = 0.0f, o2 = 0.0f, o3 = 0.0f;
            if (DK > 0) {
                float4 kv[DKP / 4], qv[DKP / 4];
#pragma unroll
                for (int i = 0; i < DKP / 4; i++) kv[i] = *(const float4*)(kt + TURN * i);
#pragma unroll
                for (int i = 0; i < DKP / 4; i++) qv[i] = *(const float4*)(qt + TURN * i);
#pragma unroll
                for (int i = 0; i < DKP / 4; i++) {
                    a0 = fmaf(S[4 * i], kv[i].x, a0); a1 = fmaf(S[4 * i + 1], kv[i].y, a1); a2 = fmaf(S[4 * i + 2], kv[i].z, a2); a3 = fmaf(S[4 * i + 3], kv[i].w, a3);
                }
                float acc = (a0 + a1) + (a2 + a3);
#pragma unroll
                for (int i = 0; i < DKP; i++) S[i] *= dec;    // while the shares meet
#pragma unroll
                for (int w = 1; w < SPLIT; w <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, w);
                const float u = beta * (vj - dec * acc);
#pragma unroll
                for (int i = 0; i < DKP / 4; i++) {
                    S[4 * i] = fmaf(kv[i].x, u, S[4 * i]); S[4 * i + 1] = fmaf(kv[i].y, u, S[4 * i + 1]);
                    S[4 * i + 2] = fmaf(kv[i].z, u, S[4 * i + 2]); S[4 * i + 3] = fmaf(kv[i].w, u, S[4 * i + 3]);
                    o0 = fmaf(S[4 * i], qv[i].x, o0); o1 = fmaf(S[4 * i + 1], qv[i].y, o1); o2 = fmaf(S[4 * i + 2], qv[i].z, o2); o3 = fmaf(S[4 * i + 3], qv[i].w, o3);
                }
                rest[tt * THREADS + threadIdx.x] = (o0 + o1) + (o2 + o3);
            } else {
                for (int i = 0; i < dk4; i += 4) {
                    const float4 kv = *(const float4*)(kt + i);
                    a0 = fmaf(Ss[i * THREADS], kv.x, a0); a1 = fmaf(Ss[(i + 1) * THREADS], kv.y, a1);
                    a2 = fmaf(Ss[(i + 2) * THREADS], kv.z, a2); a3 = fmaf(Ss[(i + 3) * THREADS], kv.w, a3);
                }
                const float u = beta * (vj - dec * ((a0 + a1) + (a2 + a3)));
                for (int i = 0; i < dk4; i += 4) {
                    const float4 kv = *(const float4*)(kt + i);
                    const float4 qv = *(const float4*)(qt + i);
                    const float s0 = fmaf(kv.x, u, dec * Ss[i * THREADS]), s1 = fmaf(kv.y, u, dec * Ss[(i + 1) * THREADS]);
                    const float s2 = fmaf(kv.z, u, dec * Ss[(i + 2) * THREADS]), s3 = fmaf(kv.w, u, dec * Ss[(i + 3) * THREADS]);
                    Ss[i * THREADS] = s0; Ss[(i + 1) * THREADS] = s1; Ss[(i + 2) * THREADS] = s2; Ss[(i + 3) * THREADS] = s3;
                    o0 = fmaf(s0, qv.x, o0); o1 = fmaf(s1, qv.y, o1); o2 = fmaf(s2, qv.z, o2); o3 = fmaf(s3, qv.w, o3);
                }
                if (live) o[((int64_t)(tb + tt) * H + h) * dv + j] = (o0 + o1) + (o2 + o3);
            }
        }
        if (DK > 0) {
            __syncthreads();
            for (int idx = threadIdx.x; idx < nt * COLS; idx += THREADS) {
                const int tt = idx / COLS, c = idx - tt * COLS;
                const float* sh = rest + tt * THREADS + c * SPLIT;
                float sum = sh[0];
#pragma unroll
                for (int w = 1; w < SPLIT; w++) sum += sh[w];
                if (j0 + c < dv) o[((int64_t)(tb + tt) * H + h) * dv + j0 + c] = sum;
            }
        }
    }
    if (live) {
        if (DK > 0) {
#pragma unroll
            for (int i = 0; i < DKP; i++) sp[(int64_t)((i >> 2) * TURN + (i & 3)) * dv] = S[i];
        } else {
            for (int i = 0; i < dk; i++) sp[(int64_t)i * dv] = Ss[i * THREADS];
        }
    }
}
extern "C" CC_API int cc_gated_delta_rule(cc_device* dev, const cc_view* q, const cc_view* k, const cc_view* v, const cc_view* a, const cc_view* b,
                                          const cc_view* a_log, const cc_view* dt_bias, const cc_view* state, int32_t H, int32_t G, int32_t dk, int32_t dv,
                                          cc_buf** out) {
    SEQ_ENTER(dev, "gated_delta_rule");
    if (!out) return cc_fail(dev, CC_ERR_ARG, "gated_delta_rule: out is NULL");
    SEQ_F32(dev, q, "gated_delta_rule q"); SEQ_F32(dev, k, "gated_delta_rule k"); SEQ_F32(dev, v, "gated_delta_rule v");
    SEQ_F32(dev, a, "gated_delta_rule a"); SEQ_F32(dev, b, "gated_delta_rule b"); SEQ_F32(dev, a_log, "gated_delta_rule a_log");
    SEQ_F32(dev, dt_bias, "gated_delta_rule dt_bias"); SEQ_F32(dev, state, "gated_delta_rule state");
    CC_REQUIRE(dev, H > 0 && G > 0 && H % G == 0 && dk > 0 && dv > 0, "gated_delta_rule: bad head counts / sizes");
    CC_REQUIRE(dev, q->ndim == 2, "gated_delta_rule: q must be [T, n_kv * dk]");
    const int64_t T = q->shape[0];
    CC_REQUIRE(dev, view_len(q) == T * G * dk && view_len(k) == T * G * dk && view_len(v) == T * H * dv && view_len(a) == T * H && view_len(b) == T * H &&
                        view_len(a_log) == H && view_len(dt_bias) == H && view_len(state) == (int64_t)H * dk * dv,
               "gated_delta_rule: operand sizes do not fit T=%lld heads=%d kv=%d dk=%d dv=%d", (long long)T, H, G, dk, dv);
    cc_buf* o = nullptr;
    int rc = cc_new_activation(dev, T * H * dv, CC_F32, false, &o);
    if (rc) return rc;
    *out = o;
    if (T == 0) return CC_OK;
    void* bdp = nullptr; size_t cls = 0;
    rc = cc_pool_alloc(dev, (size_t)T * H * 2 * 4, &bdp, &cls);
    if (rc) return rc;
    cc_launch_pdl(dev, delta_gates_kernel, (unsigned)((T * H + 255) / 256), 256, 0, fptr(a), fptr(b), fptr(a_log), fptr(dt_bias), (float*)bdp, T * H, H);
    dev->launches++;
    const bool split = dk == 32 || dk == 64 || dk == 128;
    const int threads = split ? DR_SPLIT_THREADS : DR_THREADS, cols = split ? DR_SPLIT_THREADS / (dk / 16) : DR_THREADS;
    dim3 grid((unsigned)H, (unsigned)((dv + cols - 1) / cols));
#define DR_ARGS fptr(q), fptr(k), fptr(v), (const float*)bdp, fptr(state), (float*)o->base, (int)T, H, G, dk, dv
    const int dk4 = (dk + 3) & ~3;
    // two staging buffers, and the shares of the read-out or the state
    const size_t smem = ((size_t)2 * dr_stage_floats(dk4, cols) + (size_t)(split ? DR_TB : dk4) * threads) * 4;
    if (smem > 200 * 1024) { cc_pool_free(dev, bdp, cls); return cc_fail(dev, CC_ERR_UNSUPPORTED, "gated_delta_rule: dk=%d is too large", dk); }
    cudaError_t e = cudaSuccess;
    if (smem > 48 * 1024)
        e = dk == 32    ? cudaFuncSetAttribute(delta_rule_kernel<32, 2, DR_SPLIT_THREADS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)
            : dk == 64  ? cudaFuncSetAttribute(delta_rule_kernel<64, 4, DR_SPLIT_THREADS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)
            : dk == 128 ? cudaFuncSetAttribute(delta_rule_kernel<128, 8, DR_SPLIT_THREADS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)
                        : cudaFuncSetAttribute(delta_rule_kernel<0, 1, DR_THREADS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) { cc_pool_free(dev, bdp, cls); return cc_fail(dev, CC_ERR_CUDA, "gated_delta_rule: %s", cudaGetErrorString(e)); }
    if (dk == 32) cc_launch_alone(dev, delta_rule_kernel<32, 2, DR_SPLIT_THREADS>, grid, threads, smem, DR_ARGS);
    else if (dk == 64) cc_launch_alone(dev, delta_rule_kernel<64, 4, DR_SPLIT_THREADS>, grid, threads, smem, DR_ARGS);
    else if (dk == 128) cc_launch_alone(dev, delta_rule_kernel<128, 8, DR_SPLIT_THREADS>, grid, threads, smem, DR_ARGS);
    else cc_launch_alone(dev, delta_rule_kernel<0, 1, DR_THREADS>, grid, threads, smem, DR_ARGS);
#undef DR_ARGS
    cc_pool_free(dev, bdp, cls);            // stream-ordered pool: the next user of this block runs after the kernels above
    CC_LAUNCH_CHECK(dev);
    return CC_OK;
}

// ---- sliding-window attention over a ring cache ---------------------------------------------------------------------------------------
// one warp per (token, kv head)
__global__ void kv_ring_append_kernel(float* __restrict__ kring, float* __restrict__ vring, const float* __restrict__ k, const float* __restrict__ v,
                                      const float* __restrict__ knw, float eps, int64_t pos0, int ring, int T, int G, int dk, int dv) {
    pdl_enter();
    const int64_t u = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (u >= (int64_t)T * G) return;
    const int t = (int)(u / G), g = (int)(u % G);
    const int64_t row = (pos0 + t) % ring;
    const float* kr = k + ((int64_t)t * G + g) * dk;
    float* kd = kring + (row * G + g) * dk;
    if (knw) {
        float ss = 0.0f;
        for (int c = lane; c < dk; c += 32) ss = fmaf(kr[c], kr[c], ss);
        ss = warp_sum(ss);
        const float inv = 1.0f / sqrtf(ss / (float)dk + eps);
        for (int c = lane; c < dk; c += 32) kd[c] = kr[c] * inv * knw[c];
    } else {
        for (int c = lane; c < dk; c += 32) kd[c] = kr[c];
    }
    const float* vr = v + ((int64_t)t * G + g) * dv;
    float* vd = vring + (row * G + g) * dv;
    for (int c = lane; c < dv; c += 32) vd[c] = vr[c];
}
extern "C" CC_API int cc_kv_ring_append(cc_device* dev, const cc_view* kring, const cc_view* vring, const cc_view* k, const cc_view* v, const cc_view* knw,
                                        float eps, int64_t pos0, int32_t G, int32_t dk, int32_t dv) {
    SEQ_ENTER(dev, "kv_ring_append");
    SEQ_F32(dev, kring, "kv_ring_append kring"); SEQ_F32(dev, vring, "kv_ring_append vring"); SEQ_F32(dev, k, "kv_ring_append k"); SEQ_F32(dev, v, "kv_ring_append v");
    if (knw) { SEQ_F32(dev, knw, "kv_ring_append k_norm_w"); CC_REQUIRE(dev, view_len(knw) == dk, "kv_ring_append: k_norm_w must have dk elements"); }
    CC_REQUIRE(dev, G > 0 && dk > 0 && dv > 0 && kring->ndim == 2 && k->ndim == 2 && pos0 >= 0, "kv_ring_append: bad arguments");
    const int64_t ring = kring->shape[0], T = k->shape[0];
    CC_REQUIRE(dev, view_len(kring) == ring * G * dk && view_len(vring) == ring * G * dv && view_len(k) == T * G * dk && view_len(v) == T * G * dv,
               "kv_ring_append: operand sizes do not fit kv=%d dk=%d dv=%d", G, dk, dv);
    CC_REQUIRE(dev, T <= ring, "kv_ring_append: %lld tokens do not fit a ring of %lld", (long long)T, (long long)ring);
    if (T == 0) return CC_OK;
    cc_launch_pdl(dev, kv_ring_append_kernel, (unsigned)((T * G + 7) / 8), 256, 0, fptr(kring), fptr(vring), fptr(k), fptr(v), knw ? fptr(knw) : nullptr, eps, pos0, (int)ring,
                                                                             (int)T, G, dk, dv);
    CC_LAUNCH_CHECK(dev);
    return CC_OK;
}

// A pass of many rows is two products of 32-bit operands on the tensor cores (split_gemm.cuh), tiles of 128 rows, after one kernel that cuts what many
// tiles read: queries in the order of the tiles' rows, keys and (transposed) values in the order of their positions:
//   1. WaScores: S[row][j] = (q_row . k_j) * scale - r1 ln(1 + r2 (i - j)), -inf where masked, and the largest score of each row of the tile
//   2. WaValues: out[row][d] = sum_j exp(S[row][j] - top) v[j][d] / (sum_j exp(S[row][j] - top) + sink); the weights are made while the operand is staged
// A row is one (query, head); a tile's rows are the R = n_heads / n_kv heads of one key/value head for 128 / R consecutive queries, so that keys and
// values are read once per tile and not once per (query, head).  Decoded tokens go row by row (attn_rows.cuh).
// Error against 64 bits, 512 queries of 16 heads over a window of 1024 keys of 128: 3.5e-7 of the values' size (32-bit sums on the CUDA cores: 7e-7); 58 us on
// the device where those took 204.
// The keys of a tile start at a multiple of 64 positions, a score is one sum over dk, a row's weights are added in an order that the positions of the keys
// alone decide (masked keys add an exact 0), and the value sum goes by steps of 64 positions, even ones and odd ones: a query's result does not
// depend on where the call starts or what else it carries, and differs between a prompt pass and a decoded token only by the rounding of those sums.
#define WA_ROWS 128
struct WaGeom {
    int T, H, G, R, dk, dv, window, block, ring, QT, cap;      // QT queries per tile; cap = row stride of S; block > 0: a query sees only its own block of positions
    int krs, vrs, vhs;                                  // floats between two rows of the key / value ring (vhs: between two heads' values inside a row)
    float softcap;                                      // > 0: score <- softcap * tanh(score / softcap), after the scale
    int pos0_row;                                       // pos0 % ring
    int span, dkp, dvp;                                 // keys in the cut planes ; dk and dv in whole tiles
    int64_t base0;                                      // position of the planes' first key, a multiple of 64
    int64_t pos0;
};
__host__ __device__ __forceinline__ int64_t wa_lo(const WaGeom& g, int64_t i) {
    int64_t lo = (g.window > 0 && i - g.window + 1 > 0) ? i - g.window + 1 : 0;
    if (g.block > 0) { const int64_t b = i - i % g.block; lo = b > lo ? b : lo; }
    return lo;
}

__global__ void head_rms_norm_kernel(float* __restrict__ x, const float* __restrict__ w, int64_t n_units, int hs, float eps) {
    pdl_enter();
    const int64_t u = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (u >= n_units) return;
    float* xr = x + u * hs;
    float ss = 0.0f;
    for (int c = lane; c < hs; c += 32) ss = fmaf(xr[c], xr[c], ss);
    ss = warp_sum(ss);
    const float inv = 1.0f / sqrtf(ss / (float)hs + eps);
    for (int c = lane; c < hs; c += 32) xr[c] = xr[c] * inv * w[c];
}

// what the two products share: the tile's queries and the band of keys they can see
struct WaTile {
    int steps, half, t0, tq_n, kvh, c0, qt;                   // c0: first key (from `base` on) / first value column of the tile ; qt: which tile of queries
    int band_lo, last;                                  // first and last key any of the tile's queries sees, counted from base
    int ring0;                                          // the ring's row of position base
    int at;                                             // base, counted from the first key of the cut planes
    int step0;                                          // values: the first 64-key step of this CTA (it takes every second one)
    int64_t base;                                       // a multiple of 64
};
__device__ __forceinline__ void wa_tile(const WaGeom& g, int qt, int kvh, WaTile& t) {
    t.qt = qt; t.t0 = qt * g.QT; t.kvh = kvh; t.step0 = t.half = 0;
    t.tq_n = min(g.QT, g.T - t.t0);
    const int64_t i_first = g.pos0 + t.t0, lo = wa_lo(g, i_first);
    t.base = lo & ~(int64_t)63;
    t.band_lo = (int)(lo - t.base); t.last = (int)(i_first + t.tq_n - 1 - t.base);
    t.at = (int)(t.base - g.base0);
    // the ring holds every visible position, so base lies at most ring + 62 positions before pos0
    t.ring0 = (int)((unsigned)((int)(t.base - g.pos0) + g.pos0_row + 64 + 2 * g.ring - 64 % g.ring) % (unsigned)g.ring);
}
struct WaFixed { int tq, hr; };                         // row r of a tile: its query and its head
// -> its index among the T * H rows, or -1
__device__ __forceinline__ int64_t wa_row(const WaGeom& g, const WaTile& t, WaFixed f) {
    return f.tq < t.tq_n ? (int64_t)(t.t0 + f.tq) * g.H + t.kvh * g.R + f.hr : -1;
}
// the scores of a tile of queries: groups of 4 keys x 128 rows, so that the writer (a thread per row) and the reader (likewise) both move whole lines
__device__ __forceinline__ int64_t wa_score_at(const WaTile& t, int q_tiles, int cap, int key, int r) {
    return ((int64_t)t.kvh * q_tiles + t.qt) * WA_ROWS * cap + (int64_t)(key >> 2) * (4 * WA_ROWS) + r * 4;
}
// what many tiles read, cut once into three planes of bfloat16 (split_gemm.cuh).  Blocks 0 .. row_blocks: eight elements of a query or key row per
// thread; the rest: 64 keys x 64 columns of the values, turned through shared memory.  Rows of no query, positions nobody sees and columns
// behind dk / dv are zeros.  Bound by memory: 10 bytes per element.
// ring_base0: the ring's row of position base0; lo0: the first position anybody sees
__global__ void __launch_bounds__(256) wa_cut_kernel(const float* __restrict__ q, const float* __restrict__ kring, const float* __restrict__ vring, uint8_t* __restrict__ qc,
                                                     uint8_t* __restrict__ kc, uint8_t* __restrict__ vc, WaGeom g, int q_tiles, unsigned row_blocks, int ring_base0, int lo0, int vec) {
    pdl_enter();
    const int last = (int)(g.pos0 + g.T - 1 - g.base0);       // positions are counted from base0
    const unsigned q_rows = (unsigned)(g.G * q_tiles) * WA_ROWS, k_rows = (unsigned)(g.G * g.span);
    float v[8];
    if (blockIdx.x < row_blocks) {
        const unsigned per = (unsigned)g.dkp >> 3, u = blockIdx.x * 256u + threadIdx.x;
        unsigned row = u / per;
        const int c = (int)(u - row * per) * 8;
        if (row >= q_rows + k_rows) return;
        const float* src = nullptr;
        const bool is_q = row < q_rows;
        if (is_q) {
            const unsigned r = row & (WA_ROWS - 1), tile = row / WA_ROWS, kvh = tile / (unsigned)q_tiles, tq = r / (unsigned)g.R;
            const int t = (int)(tile - kvh * q_tiles) * g.QT + (int)tq;
            if ((int)tq < g.QT && t < g.T) src = q + ((int64_t)t * g.H + kvh * g.R + (r - tq * g.R)) * g.dk;
        } else {
            row -= q_rows;
            const unsigned kvh = row / (unsigned)g.span;
            const int j = (int)(row - kvh * g.span);
            if (j >= lo0 && j <= last) src = kring + (int64_t)((unsigned)(ring_base0 + j) % (unsigned)g.ring) * g.krs + kvh * g.dk;
        }
        if (src) sg_load8(src, c, g.dk, vec, v); else sg_zero8(v);
        sg_cut((is_q ? qc : kc) + ((size_t)row * g.dkp + c) * 2, (size_t)(is_q ? q_rows : k_rows) * g.dkp * 2, v);
        return;
    }
    __shared__ float turn[64][65];
    const unsigned b = blockIdx.x - row_blocks, key_blocks = (unsigned)g.span >> 6, col_blocks = (unsigned)g.dvp >> 6, rest = b / key_blocks;
    const int j0 = (int)(b - rest * key_blocks) * 64, kvh = (int)(rest / col_blocks), d0 = (int)(rest - kvh * col_blocks) * 64, d = d0 + (threadIdx.x & 63);
    unsigned row = (unsigned)(ring_base0 + j0 + (int)(threadIdx.x >> 6)) % (unsigned)g.ring;
    const float* col = vring + (int64_t)kvh * g.vhs + d;
    float x[16];
#pragma unroll
    for (int i = 0; i < 16; i++) {
        const int j = j0 + (int)(threadIdx.x >> 6) + 4 * i;
        x[i] = j >= lo0 && j <= last && d < g.dv ? col[(int64_t)row * g.vrs] : 0.0f;
        row += 4;
        while (row >= (unsigned)g.ring) row -= (unsigned)g.ring;
    }
#pragma unroll
    for (int i = 0; i < 16; i++) turn[(threadIdx.x >> 6) + 4 * i][threadIdx.x & 63] = x[i];
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const int dd = (threadIdx.x >> 3) + 32 * i, k = (threadIdx.x & 7) * 8;
#pragma unroll
        for (int e = 0; e < 8; e++) v[e] = turn[k + e][dd];
        sg_cut(vc + (((size_t)kvh * g.dvp + d0 + dd) * g.span + j0 + k) * 2, (size_t)g.G * g.dvp * g.span * 2, v);
    }
}
// tiles: key tiles of the band (fastest), query tiles, G
struct WaScores {
    static constexpr int HALVES = 2, N = 128;
    static constexpr bool SHARED = false, A_TMA = true, SKIP_ZERO = false;
    typedef WaTile Tile;
    typedef WaFixed Fixed;
    struct Shared {};
    CUtensorMap maps[2];                                // queries [3][G][query tiles][128][dkp], keys [3][G][span][dkp]
    __device__ const void* map_a() const { return &maps[0]; }
    __device__ const void* map_b() const { return &maps[1]; }
    __device__ void at_a(const Tile& t, int s, int plane, int& x, int& y) const { x = s * 64; y = ((plane * g.G + t.kvh) * q_tiles + t.qt) * WA_ROWS; }
    __device__ void at_b(const Tile& t, int s, int plane, int& x, int& y) const { x = s * 64; y = (plane * g.G + t.kvh) * g.span + t.at + t.c0; }
    typedef const float* ARow;
    typedef const float* BCol;
    const float *q, *kring, *r1, *r2;
    float *S, *tops;                                    // tops: [G][query tiles][key tiles][4 quarters][WA_ROWS]
    WaGeom g;
    float scale;
    int key_tiles, q_tiles, vec;                        // vec: rows may be read 16 bytes at a time
    __device__ bool tile(int i, int, Tile& t) const {
        const int rest = (unsigned)i / (unsigned)key_tiles, kvh = (unsigned)rest / (unsigned)q_tiles;
        wa_tile(g, rest - kvh * q_tiles, kvh, t);
        t.c0 = (i - rest * key_tiles) * N; t.steps = (g.dk + 63) >> 6;
        return t.c0 <= t.last;
    }
    __device__ Fixed fixed(int r) const { const int tq = r / g.R; return Fixed{tq, r - tq * g.R}; }
    __device__ void setup(const Tile&, Shared&) const {}
    __device__ ARow a_row(const Tile& t, const Shared&, Fixed f, int) const {
        const int64_t row = wa_row(g, t, f);
        return row < 0 ? nullptr : q + row * g.dk;
    }
    __device__ void load_a(const Tile&, ARow a, int s, int c, float (&v)[8]) const { if (a) sg_load8(a, s * 64 + c * 8, g.dk, vec, v); else sg_zero8(v); }
    __device__ void prep_a(const Tile&, ARow&, float (&)[8]) const {}
    __device__ BCol b_col(const Tile& t, int n) const {
        const int j = t.c0 + n;
        return j < t.band_lo || j > t.last ? nullptr : kring + (int64_t)((unsigned)(t.ring0 + j) % (unsigned)g.ring) * g.krs + t.kvh * g.dk;
    }
    __device__ void load_b(const Tile&, BCol b, int s, int c, float (&v)[8]) const { if (b) sg_load8(b, s * 64 + c * 8, g.dk, vec, v); else sg_zero8(v); }
    __device__ void end_a(const Tile&, Shared&, ARow&, int, int) const {}
    __device__ void give(const Shared&, Shared&, int) const {}
    template <int COUNT>
    __device__ void emit(const Tile& t, const Shared&, Fixed f, int r, int col0, float (&v)[COUNT], float*) const {
        int lo = 0, hi = -1;                            // visible keys, counted from the first of the COUNT
        const int h = t.kvh * g.R + f.hr;
        float a1 = 0.0f, a2 = 0.0f, top = -INFINITY;
        if (f.tq < t.tq_n) {
            const int64_t i = g.pos0 + t.t0 + f.tq;
            lo = (int)(wa_lo(g, i) - t.base) - t.c0 - col0; hi = (int)(i - t.base) - t.c0 - col0;
            if (r1) { a1 = r1[h]; a2 = r2[h]; }
        }
#pragma unroll
        for (int c = 0; c < COUNT; c++) v[c] *= scale;
        if (g.softcap > 0.0f) {
#pragma unroll
            for (int c = 0; c < COUNT; c++) v[c] = g.softcap * tanhf(v[c] / g.softcap);
        }
        if (r1) {
#pragma unroll
            for (int c = 0; c < COUNT; c++) v[c] -= a1 * log1pf(a2 * (float)(hi - c));
        }
#pragma unroll
        for (int c = 0; c < COUNT; c++) {
            v[c] = c < lo || c > hi ? -INFINITY : v[c];
            top = fmaxf(top, v[c]);
        }
        float* s = S + wa_score_at(t, q_tiles, g.cap, t.c0 + col0, r);
#pragma unroll
        for (int c = 0; c < COUNT; c += 4) *(float4*)(s + c * WA_ROWS) = make_float4(v[c], v[c + 1], v[c + 2], v[c + 3]);
        tops[((((int64_t)t.kvh * q_tiles + t.qt) * key_tiles + t.c0 / N) * 4 + col0 / COUNT) * WA_ROWS + r] = top;
    }
};
// tiles: value columns (fastest), query tiles, G; the two CTAs of a cluster take the 64-key steps whose position is an even / odd multiple of 64
// sink != NULL: the denominator also holds exp(sink[head]), a key without a value whose score is sink[head] as it stands (no scale)
template <int TILE_HALVES>
struct WaValues {
    static constexpr int HALVES = TILE_HALVES, N = 64 * HALVES;
    static constexpr bool SHARED = true, A_TMA = false, SKIP_ZERO = true;
    typedef WaTile Tile;
    typedef WaFixed Fixed;
    CUtensorMap maps[1];                                // values [3][G][dvp][span]
    __device__ const void* map_a() const { return nullptr; }
    __device__ const void* map_b() const { return &maps[0]; }
    __device__ void at_a(const Tile&, int, int, int&, int&) const {}
    __device__ void at_b(const Tile& t, int s, int plane, int& x, int& y) const { x = t.at + (t.step0 + 2 * s) * 64; y = (plane * g.G + t.kvh) * g.dvp + t.c0; }
    struct Shared { float top[WA_ROWS], sum[12][WA_ROWS]; };    // sum: before the steps the quarters' largest scores (0 ..), behind them the sums of each quarter
                                                                // of the threads, of this CTA (4 ..) and of the other (8 ..)
    struct ARow { const float* s; float top, sum; };
    typedef const float* BCol;
    const float *S, *tops, *vring, *sink;
    float* o;
    WaGeom g;
    int key_tiles, q_tiles;                             // of the scores
    __device__ bool tile(int i, int rank, Tile& t) const {
        const int per = (g.dv + N - 1) / N, rest = (unsigned)i / (unsigned)per, kvh = (unsigned)rest / (unsigned)q_tiles;
        wa_tile(g, rest - kvh * q_tiles, kvh, t);
        t.c0 = (i - rest * per) * N;
        t.step0 = (int)(((t.base >> 6) & 1) ^ rank);
        t.steps = ((t.last >> 6) + 2 - t.step0) >> 1;
        t.half = (int)((((t.base >> 6) + t.step0) >> 1) & 1);      // runs by position, not by where the tile's keys begin
        return true;
    }
    __device__ Fixed fixed(int r) const { const int tq = r / g.R; return Fixed{tq, r - tq * g.R}; }
    __device__ float sink_of(const Tile& t, int r) const { return sink[t.kvh * g.R + r % g.R]; }
    // the rows' largest scores, a quarter of the threads for each quarter of a key tile
    __device__ void setup(const Tile& t, Shared& ps) const {
        const int r = threadIdx.x & 127, quarter = threadIdx.x >> 7;
        const float* p = tops + (((int64_t)t.kvh * q_tiles + t.qt) * key_tiles * 4 + quarter) * WA_ROWS + r;
        float top = -INFINITY;
#pragma unroll 8
        for (int n = 0; n <= t.last / WaScores::N; n++) top = fmaxf(top, p[n * 4 * WA_ROWS]);
        ps.sum[quarter][r] = top;
    }
    __device__ float top_of(const Tile& t, const Shared& ps, int r) const {
        float top = fmaxf(fmaxf(ps.sum[0][r], ps.sum[1][r]), fmaxf(ps.sum[2][r], ps.sum[3][r]));
        if (sink) top = fmaxf(top, sink_of(t, r));
        return top;
    }
    __device__ ARow a_row(const Tile& t, const Shared& ps, Fixed f, int r) const {
        return ARow{f.tq < t.tq_n ? S + wa_score_at(t, q_tiles, g.cap, 0, r) : nullptr, top_of(t, ps, r), 0.0f};
    }
    __device__ void load_a(const Tile& t, const ARow& a, int s, int c, float (&v)[8]) const {
        if (!a.s) { sg_zero8(v); return; }
        const float* p = a.s + ((t.step0 + 2 * s) * 16 + c * 2) * (4 * WA_ROWS);
        const float4 x = *(const float4*)p, y = *(const float4*)(p + 4 * WA_ROWS);
        v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w; v[4] = y.x; v[5] = y.y; v[6] = y.z; v[7] = y.w;
    }
    __device__ void prep_a(const Tile&, ARow& a, float (&v)[8]) const {
        if (!a.s) return;
#pragma unroll
        for (int i = 0; i < 8; i++) { v[i] = expf(v[i] - a.top); a.sum += v[i]; }
    }
    __device__ BCol b_col(const Tile& t, int n) const { return t.c0 + n < g.dv ? vring + t.kvh * g.vhs + t.c0 + n : nullptr; }
    __device__ void load_b(const Tile& t, BCol b, int s, int c, float (&v)[8]) const {
        const int k = (t.step0 + 2 * s) * 64 + c * 8;
        unsigned row = (unsigned)(t.ring0 + k);
        while (row >= (unsigned)g.ring) row -= (unsigned)g.ring;
        if (b && k >= t.band_lo && k + 7 <= t.last && row + 8 <= (unsigned)g.ring) {
            const float* at = b + (int64_t)row * g.vrs;
#pragma unroll
            for (int i = 0; i < 8; i++) { v[i] = *at; at += g.vrs; }
            return;
        }
#pragma unroll
        for (int i = 0; i < 8; i++) {
            v[i] = b && k + i >= t.band_lo && k + i <= t.last ? b[(int64_t)row * g.vrs] : 0.0f;
            if (++row == (unsigned)g.ring) row = 0;
        }
    }
    __device__ void end_a(const Tile&, Shared& ps, const ARow& a, int r, int part) const {
        ps.sum[4 + part][r] = a.sum;
        if (part == 0) ps.top[r] = a.top;
    }
    // a CTA's sums of weights to the other
    __device__ void give(const Shared& mine, Shared& theirs, int tid) const { theirs.sum[8 + (tid >> 7)][tid & 127] = mine.sum[4 + (tid >> 7)][tid & 127]; }
    template <int COUNT>
    __device__ void emit(const Tile& t, const Shared& ps, Fixed f, int r, int col0, float (&v)[COUNT], float* buf) const {
        float a = 0.0f, b = 0.0f;
#pragma unroll
        for (int i = 0; i < 4; i++) { a += ps.sum[4 + i][r]; b += ps.sum[8 + i][r]; }
        float total = a + b;                            // of the two CTAs, the same number in both
        if (sink) total += expf(sink_of(t, r) - ps.top[r]);
        const float inv = 1.0f / total;
#pragma unroll
        for (int c = 0; c < COUNT; c++) v[c] *= inv;
        const int64_t row = wa_row(g, t, f);
        sg_store_rows<COUNT>(buf, row < 0 ? nullptr : o + row * g.dv + t.c0 + col0, g.dv - t.c0 - col0, g.dv % 4 == 0, v);
    }
};
#include "attn_rows.cuh"
// what a call's two ways share
struct WaCall {
    float* q;
    const float *k, *v, *r1, *r2, *sink;
    float *o, scale;
    int64_t last, oldest, reach;                        // last position; first one anybody sees; the most keys one query sees
};
// few rows: keys spread over the whole device
static int wa_by_rows(cc_device* dev, const WaGeom& g, const WaCall& c) {
    ArArgs A{};
    A.q = c.q; A.k = c.k; A.v = c.v; A.r1 = c.r1; A.r2 = c.r2; A.sink = c.sink; A.out = c.o; A.scale = c.scale;
    return attn_rows(dev, g, A, (int)c.reach);
}
// many rows: key/value heads in equal groups, so that the workspace -- scores and cut planes of a group -- is at most twice what the scores of all heads take
// or WA_WORKSPACE, whichever is more (one head at least).  *room: false when the device had none and nothing was launched
#define WA_WORKSPACE ((size_t)512 << 20)
static int wa_by_tiles(cc_device* dev, WaGeom g, const WaCall& c, bool* room) {
    const int G = g.G, q_tiles = (g.T + g.QT - 1) / g.QT, vtile = g.dv > 64 ? 128 : 64;
    // keys a query tile can see, counted from the multiple of 64 below the first of them
    const int64_t band = c.reach - 1 + g.QT + 63, band_max = band < c.last + 64 ? band : c.last + 64;
    const int key_tiles = (int)((band_max + WaScores::N - 1) / WaScores::N);
    g.cap = key_tiles * WaScores::N;
    g.base0 = c.oldest & ~(int64_t)63;
    g.span = (int)((c.last - g.base0 + 64) & ~(int64_t)63) + 64;              // in whole steps, and one more: a tile of 128 keys may start at any step
    g.dkp = (g.dk + 63) & ~63; g.dvp = (g.dv + vtile - 1) / vtile * vtile;
    // of one key/value head; every part is a multiple of 512 bytes
    const size_t q_rows = (size_t)q_tiles * WA_ROWS, scores = q_rows * g.cap * 4, tops = (size_t)q_tiles * key_tiles * 4 * WA_ROWS * 4;
    const size_t qc = 3 * q_rows * g.dkp * 2, kc = 3 * (size_t)g.span * g.dkp * 2, vc = 3 * (size_t)g.dvp * g.span * 2, one = scores + tops + qc + kc + vc;
    const size_t scores_twice = 2 * (size_t)g.T * g.H * c.reach * 4, most = scores_twice > WA_WORKSPACE ? scores_twice : WA_WORKSPACE;
    int groups = (int)((G * one + most - 1) / most);
    if (groups > G) groups = G;
    void* S = nullptr; size_t cls = 0;
    int rc, n = 0;
    for (;; groups = groups * 2 < G ? groups * 2 : G) {
        n = (G + groups - 1) / groups;
        if (3 * n * (q_rows + g.span) * (g.dkp / 8) >= (size_t)1 << 31) rc = cc_fail(dev, CC_ERR_UNSUPPORTED, "window_attention: too many rows");      // 32-bit indices
        else rc = cc_pool_alloc(dev, n * one, &S, &cls);
        if (rc == CC_OK) break;
        cudaGetLastError();                                  // it has been taken note of
        if (n == 1) { *room = false; return rc; }
    }
    uint8_t *base = (uint8_t*)S, *qp3 = base + n * (scores + tops), *kp3 = qp3 + n * qc, *vp3 = kp3 + n * kc;
    WaScores ws{};
    ws.S = (float*)base; ws.tops = (float*)(base + n * scores); ws.scale = c.scale; ws.key_tiles = key_tiles; ws.q_tiles = q_tiles;
    ws.vec = g.dk % 4 == 0 && (((uintptr_t)c.q | (uintptr_t)c.k) & 15) == 0;
    for (int g0 = 0; g0 < G && rc == CC_OK; g0 += n) {
        const int h0 = g0 * g.R;
        g.G = G - g0 < n ? G - g0 : n;
        const float* v = c.v + (int64_t)g0 * g.vhs;
        ws.q = c.q + (int64_t)h0 * g.dk; ws.kring = c.k + (int64_t)g0 * g.dk; ws.r1 = c.r1 ? c.r1 + h0 : nullptr; ws.r2 = c.r2 ? c.r2 + h0 : nullptr; ws.g = g;
        const size_t rows = (size_t)g.G * q_rows;
        const int64_t row_blocks = ((int64_t)(rows + (size_t)g.G * g.span) * (g.dkp >> 3) + 255) / 256, blocks = row_blocks + (int64_t)(g.span >> 6) * (g.dvp >> 6) * g.G;
        CUtensorMap vmap;
        rc = cc_make_tmap_bf16(dev, &ws.maps[0], qp3, 3 * (int64_t)rows, g.dkp, WA_ROWS);
        if (rc == CC_OK) rc = cc_make_tmap_bf16(dev, &ws.maps[1], kp3, (int64_t)3 * g.G * g.span, g.dkp, WaScores::N);
        if (rc == CC_OK) rc = cc_make_tmap_bf16(dev, &vmap, vp3, (int64_t)3 * g.G * g.dvp, g.span, vtile);
        if (rc == CC_OK) {
            cc_launch_pdl(dev, wa_cut_kernel, (unsigned)blocks, 256, 0, ws.q, ws.kring, v, qp3, kp3, vp3, g, q_tiles, (unsigned)row_blocks, (int)(g.base0 % g.ring), (int)(c.oldest - g.base0), ws.vec);
            dev->launches++;
            rc = sg_launch(dev, ws, (int64_t)key_tiles * q_tiles * g.G);
        }
        auto values = [&](auto wv) {
            wv.maps[0] = vmap; wv.S = ws.S; wv.tops = ws.tops; wv.vring = v; wv.sink = c.sink ? c.sink + h0 : nullptr; wv.o = c.o + (int64_t)h0 * g.dv; wv.g = g;
            wv.key_tiles = key_tiles; wv.q_tiles = q_tiles;
            return sg_launch<decltype(wv), true>(dev, wv, (int64_t)(g.dvp / vtile) * q_tiles * g.G);
        };
        if (rc == CC_OK) rc = vtile == 128 ? values(WaValues<2>{}) : values(WaValues<1>{});
    }
    cc_pool_free(dev, S, cls);
    return rc;
}
static int masked_attention_impl(cc_device* dev, const cc_view* q, const cc_view* qnw, float eps, const cc_view* kring, const cc_view* vring, int64_t pos0, int32_t H, int32_t G,
                                 int32_t dk, int32_t dv, int32_t window, int32_t block, float scale, const cc_view* r1, const cc_view* r2, const cc_view* sink, cc_buf** out,
                                 float softcap = 0.0f) {
    SEQ_ENTER(dev, "window_attention");
    if (!out) return cc_fail(dev, CC_ERR_ARG, "window_attention: out is NULL");
    SEQ_F32(dev, q, "window_attention q"); SEQ_F32(dev, kring, "window_attention kring");
    if (vring) SEQ_F32(dev, vring, "window_attention vring");
    if (sink) { SEQ_F32(dev, sink, "window_attention sink"); CC_REQUIRE(dev, view_len(sink) == H, "window_attention: sink must have one number per head"); }
    if (qnw) { SEQ_F32(dev, qnw, "window_attention q_norm_w"); CC_REQUIRE(dev, view_len(qnw) == dk, "window_attention: q_norm_w must have dk elements"); }
    CC_REQUIRE(dev, (r1 == nullptr) == (r2 == nullptr), "window_attention: r1 and r2 come together");
    if (r1) {
        SEQ_F32(dev, r1, "window_attention r1"); SEQ_F32(dev, r2, "window_attention r2");
        CC_REQUIRE(dev, view_len(r1) == H && view_len(r2) == H, "window_attention: r1 / r2 must have one number per head");
    }
    CC_REQUIRE(dev, H > 0 && G > 0 && H % G == 0 && dk > 0 && dv > 0 && q->ndim == 2 && kring->ndim == 2 && pos0 >= 0, "window_attention: bad arguments");
    const int64_t T = q->shape[0], ring = kring->shape[0];
    CC_REQUIRE(dev, view_len(q) == T * H * dk && view_len(kring) == ring * G * dk && (vring ? view_len(vring) == ring * G * dv : dv <= dk),
               "window_attention: operand sizes do not fit heads=%d kv=%d dk=%d dv=%d", H, G, dk, dv);
    const float* vptr = vring ? fptr(vring) : fptr(kring);            // no value ring: a key row's first dv columns are its value
    // the oldest row the first query needs must not have been overwritten by the newest row of this call
    const int64_t last = pos0 + T - 1;
    WaGeom g;
    g.window = window; g.block = block; g.softcap = softcap;
    const int64_t oldest = wa_lo(g, pos0);
    CC_REQUIRE(dev, T == 0 || last - oldest + 1 <= ring, "window_attention: positions %lld..%lld with window %d, block %d need more than the ring's %lld rows",
               (long long)pos0, (long long)last, window, block, (long long)ring);
    cc_buf* o = nullptr;
    int rc = cc_new_activation(dev, T * H * dv, CC_F32, false, &o);
    if (rc) return rc;
    *out = o;
    if (T == 0) return CC_OK;
    // the most keys one query can see
    int64_t reach = last + 1;
    if (window > 0 && window < reach) reach = window;
    if (block > 0 && block < reach) reach = block;
    const int R = H / G;
    CC_REQUIRE(dev, R <= 64, "window_attention: %d query heads per key/value head (at most %d)", R, 64);
    g.T = (int)T; g.H = H; g.G = G; g.R = R; g.dk = dk; g.dv = dv; g.ring = (int)ring; g.QT = WA_ROWS / R; g.pos0 = pos0; g.pos0_row = (int)(pos0 % ring);
    g.krs = G * dk; g.vrs = vring ? G * dv : G * dk; g.vhs = vring ? dv : dk;
    const WaCall c = {fptr(q), fptr(kring), vptr, r1 ? fptr(r1) : nullptr, r2 ? fptr(r2) : nullptr, sink ? fptr(sink) : nullptr, (float*)o->base, scale, last, oldest, reach};
    // Row by row the cache is read once per query and 16 heads of a key head, and a key takes about 2e-7 us for each of
    //     cost = T * (key heads x blocks of heads) * (dk + dv in whole 128s + 128 for the sums across lanes) * (2, 3, 4, 7 or 12 for up to 1, 2, 4, 8 or 16 heads);
    // a tile's work is the same up to 128 rows, 20 to 30 us and 0.012 us a key.  More than 64 rows are tiles whatever they cost (one or two queries of few blocks of heads
    // aside): the portions of a prompt that have more take the same way and a query its bits with them, however the prompt is cut.  Portions of 64 rows or fewer may take the other one,
    // by how many queries they have and how long the cache is, and the two ways' bits differ.  us by rows / by tiles over 300, 2000, 4000, 16000 keys, heads on key heads x queries:
    // 16 on 16 x 4 13 / 27, 30 / 57, 50 / 103, 138 / 352 ; 8 on 1 (latent, 576) x 8 18 / 31, 41 / 51, 70 / 73, 222 / 223 ; 4 on 1 (latent) x 16 22 / 31, 52 / 52, 87 / 73, 229 / 223 ;
    // 1 on 1 (latent) x 32 19 / 31, 57 / 51, 104 / 73, 275 / 222 ; 128 on 128 (192, 128) x 2 34 / 79, 120 / 319, 209 / 632
    const bool can_rows = T <= 65535 && (int64_t)(R < 8 ? R : 8) * dk * 4 <= 160 * 1024;
    const int64_t cost = T * G * ((R + 15) / 16) * ((((int64_t)dk + 127) & ~127) + (((int64_t)dv + 127) & ~127) + 128) * (R > 8 ? 12 : R > 4 ? 7 : R > 2 ? 4 : R + 1);
    const bool few_rows = can_rows && ((T * H <= 64 && cost <= 72000 + 12000000 / reach) || (T <= 2 && T * ((R + 7) / 8) <= 4) || ring >= (1 << 30));
    if (qnw) {             // the query norm, in place: q is this call's private projection output in every caller of the runner; a caller that
                           // needs its q untouched passes a copy
        cc_launch_pdl(dev, head_rms_norm_kernel, (unsigned)((T * H + 7) / 8), 256, 0, c.q, fptr(qnw), T * H, dk, eps);
        dev->launches++;
    }
    if (few_rows) return wa_by_rows(dev, g, c);
    CC_REQUIRE(dev, ring < (1 << 30), "window_attention: too many rows");
    bool room = true;
    rc = wa_by_tiles(dev, g, c, &room);
    return !room && can_rows ? wa_by_rows(dev, g, c) : rc;
}
extern "C" CC_API int cc_window_attention_sink(cc_device* dev, const cc_view* q, const cc_view* qnw, float eps, const cc_view* kring, const cc_view* vring, int64_t pos0,
                                               int32_t H, int32_t G, int32_t dk, int32_t dv, int32_t window, float scale, const cc_view* r1, const cc_view* r2,
                                               const cc_view* sink, cc_buf** out) {
    return masked_attention_impl(dev, q, qnw, eps, kring, vring, pos0, H, G, dk, dv, window, 0, scale, r1, r2, sink, out);
}
extern "C" CC_API int cc_masked_attention(cc_device* dev, const cc_view* q, const cc_view* kring, const cc_view* vring, int64_t pos0, int32_t H, int32_t G, int32_t dk, int32_t dv,
                                          int32_t window, int32_t block, float scale, const cc_view* sink, cc_buf** out) {
    return masked_attention_impl(dev, q, nullptr, 0.0f, kring, vring, pos0, H, G, dk, dv, window, block, scale, nullptr, nullptr, sink, out);
}
extern "C" CC_API int cc_masked_attention_capped(cc_device* dev, const cc_view* q, const cc_view* kring, const cc_view* vring, int64_t pos0, int32_t H, int32_t G, int32_t dk,
                                                 int32_t dv, int32_t window, int32_t block, float scale, float softcap, const cc_view* sink, cc_buf** out) {
    return masked_attention_impl(dev, q, nullptr, 0.0f, kring, vring, pos0, H, G, dk, dv, window, block, scale, nullptr, nullptr, sink, out, softcap);
}
extern "C" CC_API int cc_window_attention(cc_device* dev, const cc_view* q, const cc_view* qnw, float eps, const cc_view* kring, const cc_view* vring, int64_t pos0,
                                          int32_t H, int32_t G, int32_t dk, int32_t dv, int32_t window, float scale, const cc_view* r1, const cc_view* r2,
                                          cc_buf** out) {
    if (dev && !vring) return cc_fail(dev, CC_ERR_ARG, "window_attention: vring is NULL");
    return cc_window_attention_sink(dev, q, qnw, eps, kring, vring, pos0, H, G, dk, dv, window, scale, r1, r2, nullptr, out);
}

// ---- RMS norm in groups ----------------------------------------------------------------------------------------------------------------
// one warp per (row, group): the units are consecutive in memory, unit u covers x[u * gs, (u + 1) * gs)
__global__ void group_rms_norm_kernel(float* __restrict__ dst, const float* __restrict__ x, const float* __restrict__ w, int64_t n_units, int groups, int gs, float eps) {
    pdl_enter();
    const int64_t u = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (u >= n_units) return;
    const float* xr = x + u * gs;
    const float* wr = w + (u % groups) * gs;
    float ss = 0.0f;
    for (int c = lane; c < gs; c += 32) ss = fmaf(xr[c], xr[c], ss);
    ss = warp_sum(ss);
    const float inv = 1.0f / sqrtf(ss / (float)gs + eps);
    float* dr = dst + u * gs;
    for (int c = lane; c < gs; c += 32) dr[c] = xr[c] * inv * wr[c];
}
// a wide group: one CTA per (row, group), the order of rms_norm_gain_wide_kernel
__global__ void __launch_bounds__(RNG_THREADS) group_rms_norm_wide_kernel(float* __restrict__ dst, const float* __restrict__ x, const float* __restrict__ w, int groups, int gs, float eps) {
    pdl_enter();
    __shared__ float red[RNG_THREADS / 32];
    const int64_t u = blockIdx.x;
    const float* xr = x + u * gs;
    const float* wr = w + (u % groups) * gs;
    float ss = 0.0f;
    for (int c = threadIdx.x; c < gs; c += RNG_THREADS) ss = fmaf(xr[c], xr[c], ss);
    ss = warp_sum(ss);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
    __syncthreads();
    float tot = 0.0f;
#pragma unroll
    for (int i = 0; i < RNG_THREADS / 32; i++) tot += red[i];
    const float inv = 1.0f / sqrtf(tot / (float)gs + eps);
    float* dr = dst + u * gs;
    for (int c = threadIdx.x; c < gs; c += RNG_THREADS) dr[c] = xr[c] * inv * wr[c];
}
extern "C" CC_API int cc_group_rms_norm(cc_device* dev, const cc_view* dst, const cc_view* x, const cc_view* w, int32_t groups, float eps) {
    SEQ_ENTER(dev, "group_rms_norm");
    SEQ_F32(dev, dst, "group_rms_norm dst"); SEQ_F32(dev, x, "group_rms_norm x"); SEQ_F32(dev, w, "group_rms_norm w");
    CC_REQUIRE(dev, x->ndim == 2 && dst->ndim == 2 && dst->shape[0] == x->shape[0] && dst->shape[1] == x->shape[1], "group_rms_norm: dst and x must be [rows, cols]");
    const int64_t rows = x->shape[0], cols = x->shape[1];
    CC_REQUIRE(dev, groups >= 1 && cols % groups == 0 && view_len(w) == cols, "group_rms_norm: %lld columns, %d groups, %lld weights", (long long)cols, groups, (long long)view_len(w));
    if (rows == 0) return CC_OK;
    const int64_t units = rows * groups;
    if (cols / groups >= 512) cc_launch_pdl(dev, group_rms_norm_wide_kernel, (unsigned)units, RNG_THREADS, 0, fptr(dst), fptr(x), fptr(w), groups, (int)(cols / groups), eps);
    else cc_launch_pdl(dev, group_rms_norm_kernel, (unsigned)((units + 7) / 8), 256, 0, fptr(dst), fptr(x), fptr(w), units, groups, (int)(cols / groups), eps);
    CC_LAUNCH_CHECK(dev);
    return CC_OK;
}

// ---- layer norm with weight and bias ------------------------------------------------------------------------------------------------------
// one CTA per row (layer_norm.cuh)
#define LN_THREADS 256
__global__ void __launch_bounds__(LN_THREADS) layer_norm_kernel(float* dst, const float* x, const float* __restrict__ w, const float* __restrict__ b, int cols, float eps) {
    pdl_enter();
    __shared__ float red[LN_THREADS / 32];
    float* dr = dst + (int64_t)blockIdx.x * cols;
    layer_norm_row<LN_THREADS>(x + (int64_t)blockIdx.x * cols, w, b, cols, eps, red, [&](int c, float v) { dr[c] = v; });
}
extern "C" CC_API int cc_layer_norm(cc_device* dev, const cc_view* dst, const cc_view* x, const cc_view* w, const cc_view* b, float eps) {
    SEQ_ENTER(dev, "layer_norm");
    SEQ_F32(dev, dst, "layer_norm dst"); SEQ_F32(dev, x, "layer_norm x"); SEQ_F32(dev, w, "layer_norm w");
    if (b) SEQ_F32(dev, b, "layer_norm b");
    CC_REQUIRE(dev, x->ndim == 2 && dst->ndim == 2 && dst->shape[0] == x->shape[0] && dst->shape[1] == x->shape[1], "layer_norm: dst and x must be [rows, cols]");
    const int64_t rows = x->shape[0], cols = x->shape[1];
    CC_REQUIRE(dev, cols >= 1 && view_len(w) == cols && (!b || view_len(b) == cols), "layer_norm: %lld columns need as many weights (and biases)", (long long)cols);
    if (rows == 0) return CC_OK;
    cc_launch_pdl(dev, layer_norm_kernel, (unsigned)rows, LN_THREADS, 0, fptr(dst), fptr(x), fptr(w), b ? fptr(b) : nullptr, (int)cols, eps);
    CC_LAUNCH_CHECK(dev);
    return CC_OK;
}

// the gate first, then the norm.  One warp per (row, group), or one CTA of GGN_THREADS threads when a group is wide (a single warp would walk
// it in many dependent trips to memory).  Either way the gated value is written once, its squares are summed in an order that depends on
// the group's size alone (lane- or thread-strided partial sums, the butterfly, then the warps' sums in warp order), and the value is scaled.
#define GGN_THREADS 256
__global__ void gated_group_rms_norm_kernel(float* dst, const float* x, const float* __restrict__ gate, const float* __restrict__ w, int64_t n_units,
                                            int groups, int gs, float eps, int act, int64_t grs) {
    pdl_enter();
    const int64_t u = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (u >= n_units) return;
    const float* xr = x + u * gs;
    const float* gr = gate + (u / groups) * grs + (u % groups) * gs;
    const float* wr = w + (u % groups) * gs;
    float* dr = dst + u * gs;
    float ss = 0.0f;
    for (int c = lane; c < gs; c += 32) { const float v = xr[c] * seq_act(gr[c], act); dr[c] = v; ss = fmaf(v, v, ss); }
    ss = warp_sum(ss);
    const float inv = 1.0f / sqrtf(ss / (float)gs + eps);
    for (int c = lane; c < gs; c += 32) dr[c] = dr[c] * inv * wr[c];
}
__global__ void __launch_bounds__(GGN_THREADS) gated_group_rms_norm_wide_kernel(float* dst, const float* x, const float* __restrict__ gate,
                                                                                const float* __restrict__ w, int groups, int gs, float eps, int act, int64_t grs) {
    pdl_enter();
    __shared__ float red[GGN_THREADS / 32];
    const int64_t u = blockIdx.x;
    const float* xr = x + u * gs;
    const float* gr = gate + (u / groups) * grs + (u % groups) * gs;
    const float* wr = w + (u % groups) * gs;
    float* dr = dst + u * gs;
    float ss = 0.0f;
    for (int c = threadIdx.x; c < gs; c += GGN_THREADS) { const float v = xr[c] * seq_act(gr[c], act); dr[c] = v; ss = fmaf(v, v, ss); }
    ss = warp_sum(ss);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
    __syncthreads();
    float tot = 0.0f;
#pragma unroll
    for (int i = 0; i < GGN_THREADS / 32; i++) tot += red[i];
    const float inv = 1.0f / sqrtf(tot / (float)gs + eps);
    for (int c = threadIdx.x; c < gs; c += GGN_THREADS) dr[c] = dr[c] * inv * wr[c];
}
extern "C" CC_API int cc_gated_group_rms_norm(cc_device* dev, const cc_view* dst, const cc_view* x, const cc_view* gate, const cc_view* w, int32_t groups, float eps,
                                              int32_t gate_act) {
    SEQ_ENTER(dev, "gated_group_rms_norm");
    SEQ_F32(dev, dst, "gated_group_rms_norm dst"); SEQ_F32(dev, x, "gated_group_rms_norm x"); SEQ_ROWS(dev, gate, "gated_group_rms_norm gate"); SEQ_F32(dev, w, "gated_group_rms_norm w");
    CC_REQUIRE(dev, x->ndim == 2 && dst->ndim == 2 && dst->shape[0] == x->shape[0] && dst->shape[1] == x->shape[1] && gate->shape[0] == x->shape[0] && gate->shape[1] == x->shape[1],
               "gated_group_rms_norm: dst, x and gate must be [rows, cols]");
    const int64_t grs = gate->strides[0];
    const int64_t rows = x->shape[0], cols = x->shape[1];
    CC_REQUIRE(dev, groups >= 1 && cols % groups == 0 && view_len(w) == cols, "gated_group_rms_norm: %lld columns, %d groups, %lld weights", (long long)cols, groups,
               (long long)view_len(w));
    if (rows == 0) return CC_OK;
    const int64_t units = rows * groups;
    const int gs = (int)(cols / groups);
    if (gs >= 512) cc_launch_pdl(dev, gated_group_rms_norm_wide_kernel, (unsigned)units, GGN_THREADS, 0, fptr(dst), fptr(x), fptr(gate), fptr(w), groups, gs, eps, gate_act, grs);
    else cc_launch_pdl(dev, gated_group_rms_norm_kernel, (unsigned)((units + 7) / 8), 256, 0, fptr(dst), fptr(x), fptr(gate), fptr(w), units, groups, gs, eps, gate_act, grs);
    CC_LAUNCH_CHECK(dev);
    return CC_OK;
}

// ---- rotary positions from a frequency table, neighbouring coordinates paired -------------------------------------------------------------
// the angle is the 32-bit product of the position and the pair's frequency; cosf / sinf are the accurate library functions
__device__ __forceinline__ void rotate_pair(float u, float v, float pos, float f, float mag, float& ou, float& ov) {
    const float a = pos * f;
    const float c = cosf(a) * mag, s = sinf(a) * mag;
    ou = u * c - v * s;
    ov = v * c + u * s;
}
// one thread per (token, head, pair)
// pair i of a head is the columns off + i * step and off + i * step + gap: (step, gap) = (2, 1) pairs neighbours, (1, half) pairs the two
// halves of the rotated columns
__global__ void rope_pairs_kernel(float* x, const float* __restrict__ freq, int64_t n, int heads, int hs, int off, int half, float mag, int64_t pos0, int step, int gap,
                                  float* x2) {
    pdl_enter();
    int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (x2 ? 2 * n : n)) return;
    if (idx >= n) { idx -= n; x = x2; }                              // a second tensor of the same shape rides along
    const int i = (int)(idx % half);
    const int64_t th = idx / half;                                   // token * heads + head
    float* p = x + th * hs + off + step * i;
    float ou, ov;
    rotate_pair(p[0], p[gap], (float)(pos0 + th / heads), freq[i], mag, ou, ov);
    p[0] = ou; p[gap] = ov;
}
static int rope_table_impl(cc_device* dev, const cc_view* x, int32_t n_heads, int32_t head_size, int32_t offset, const cc_view* freq, float mag, int64_t pos0, bool halves,
                           const cc_view* x2 = nullptr);
extern "C" CC_API int cc_rope_pairs(cc_device* dev, const cc_view* x, int32_t n_heads, int32_t head_size, int32_t offset, const cc_view* freq, float mag, int64_t pos0) {
    return rope_table_impl(dev, x, n_heads, head_size, offset, freq, mag, pos0, false);
}
extern "C" CC_API int cc_rope_halves(cc_device* dev, const cc_view* x, int32_t n_heads, int32_t head_size, int32_t offset, const cc_view* freq, float mag, int64_t pos0) {
    return rope_table_impl(dev, x, n_heads, head_size, offset, freq, mag, pos0, true);
}
extern "C" CC_API int cc_rope_halves_two(cc_device* dev, const cc_view* x1, const cc_view* x2, int32_t n_heads, int32_t head_size, int32_t offset, const cc_view* freq, float mag,
                                         int64_t pos0) {
    if (dev && !x2) return cc_fail(dev, CC_ERR_ARG, "rope_halves_two: the second tensor is NULL");
    return rope_table_impl(dev, x1, n_heads, head_size, offset, freq, mag, pos0, true, x2);
}
static int rope_table_impl(cc_device* dev, const cc_view* x, int32_t n_heads, int32_t head_size, int32_t offset, const cc_view* freq, float mag, int64_t pos0, bool halves,
                           const cc_view* x2) {
    SEQ_ENTER(dev, "rope_pairs");
    if (x2) { SEQ_F32(dev, x2, "rope_pairs second tensor"); CC_REQUIRE(dev, x2->ndim == 2 && x->ndim == 2 && x2->shape[0] == x->shape[0] && x2->shape[1] == x->shape[1], "rope_pairs: the two tensors differ in shape"); }
    SEQ_F32(dev, x, "rope_pairs x"); SEQ_F32(dev, freq, "rope_pairs freq");
    const int64_t half = view_len(freq);
    CC_REQUIRE(dev, x->ndim == 2 && n_heads > 0 && head_size > 0 && x->shape[1] == (int64_t)n_heads * head_size && offset >= 0 && offset + 2 * half <= head_size && pos0 >= 0,
               "rope_pairs: %lld pairs at column %d do not fit heads of %d", (long long)half, offset, head_size);
    const int64_t n = x->shape[0] * n_heads * half;
    if (n == 0) return CC_OK;
    const int64_t items = x2 ? 2 * n : n;
    cc_launch_pdl(dev, rope_pairs_kernel, (unsigned)((items + 255) / 256), 256, 0, fptr(x), fptr(freq), n, n_heads, head_size, offset, (int)half, mag, pos0, halves ? 1 : 2,
                                                                                halves ? (int)half : 1, x2 ? fptr(x2) : nullptr);
    CC_LAUNCH_CHECK(dev);
    return CC_OK;
}

// ---- queries and keys from projection to cache in one pass ---------------------------------------------------------------------------------
struct QkPrepArgs {
    const float *q, *k, *v;                                 // row t of the raw operands at q + t * qrs, k + t * krs, v + t * vrs
    float *qo, *kring, *vring;                              // qo: [T, H * dk], may be q itself
    int64_t qrs, krs, vrs;
    const float *qw, *kw, *freq;
    int H, G, dk, dv, ring, norm, half, step, gap, off;      // pair i of a head: columns off + i * step and off + i * step + gap
    float eps, mag;
    int64_t pos0;
};
#define QKP_THREADS 256
// grid (tokens, blocks of heads); a norm over the whole projection takes one block, whose sums (thread-strided, butterfly, the warps' sums in warp order) come
// first.  A warp takes a head: its inverse root mean square (lane-strided sum, butterfly), then every element once, a rotated pair by the lane of its
// first column, which reads both raw values and writes both results, so q may be overwritten in place.  (With the heads' factors passed through shared memory and an
// integer division per element: 4.9 us a decoded token and 8.5 us for 512 rows of 8 + 2 heads of 128; now 3.1 and 5.2.)
__global__ void __launch_bounds__(QKP_THREADS) qk_prepare_kernel(QkPrepArgs a) {
    pdl_enter();
    __shared__ float red[QKP_THREADS / 32];
    float inv[2];
    const int t = blockIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int units_all = a.H + a.G, per_block = (units_all + gridDim.y - 1) / gridDim.y;
    const int u0 = min(units_all, (int)blockIdx.y * per_block), u1 = min(units_all, u0 + per_block);       // this CTA's heads: queries', then keys'
    const float* qr = a.q + t * a.qrs;
    const float* kr = a.k + t * a.krs;
    float* qo = a.qo + (int64_t)t * a.H * a.dk;
    if (a.norm == CC_QK_NORM_ROW) {
        for (int side = 0; side < 2; side++) {
            const float* src = side ? kr : qr;
            const int n = (side ? a.G : a.H) * a.dk;
            float ss = 0.0f;
            for (int c = threadIdx.x; c < n; c += QKP_THREADS) ss = fmaf(src[c], src[c], ss);
            ss = warp_sum(ss);
            __syncthreads();
            if (lane == 0) red[w] = ss;
            __syncthreads();
            float tot = 0.0f;
#pragma unroll
            for (int i = 0; i < QKP_THREADS / 32; i++) tot += red[i];
            inv[side] = 1.0f / sqrtf(tot / (float)n + a.eps);
        }
        __syncthreads();                             // all raw values have been read for the sums
    }
    const int64_t row = (a.pos0 + t) % a.ring;
    const float pos = (float)(a.pos0 + t);
    for (int u = u0 + w; u < u1; u += QKP_THREADS / 32) {
        const bool is_q = u < a.H;
        const int ul = is_q ? u : u - a.H;
        const float* src = is_q ? qr + u * a.dk : kr + ul * a.dk;
        float* dst = is_q ? qo + u * a.dk : a.kring + (row * a.G + ul) * a.dk;
        const float* wt = is_q ? a.qw : a.kw;
        if (wt && a.norm == CC_QK_NORM_ROW) wt += ul * a.dk;
        float f = a.norm == CC_QK_NORM_ROW ? inv[is_q ? 0 : 1] : 1.0f;
        if (a.norm == CC_QK_NORM_HEAD) {
            float ss = 0.0f;
#pragma unroll 4
            for (int c = lane; c < a.dk; c += 32) ss = fmaf(src[c], src[c], ss);
            ss = warp_sum(ss);
            f = 1.0f / sqrtf(ss / (float)a.dk + a.eps);
        }
        // a rotated pair by the lane of its first column
        const int first = a.half > 0 ? a.off : a.dk, behind = a.half > 0 ? a.off + 2 * a.half : a.dk;
        for (int i = lane; i < a.half; i += 32) {
            const int c = a.off + a.step * i, c1 = c + a.gap;
            const float x0 = wt ? src[c] * f * wt[c] : src[c] * f, x1 = wt ? src[c1] * f * wt[c1] : src[c1] * f;
            float o0, o1;
            rotate_pair(x0, x1, pos, a.freq[i], a.mag, o0, o1);
            dst[c] = o0; dst[c1] = o1;
        }
        for (int c = lane; c < first; c += 32) dst[c] = wt ? src[c] * f * wt[c] : src[c] * f;
        for (int c = behind + lane; c < a.dk; c += 32) dst[c] = wt ? src[c] * f * wt[c] : src[c] * f;
    }
    const float* vr = a.v + t * a.vrs;
    float* vd = a.vring + row * a.G * a.dv;
    for (int c = blockIdx.y * QKP_THREADS + threadIdx.x; c < a.G * a.dv; c += gridDim.y * QKP_THREADS) vd[c] = vr[c];
}
static int qk_prepare_impl(cc_device* dev, QkPrepArgs a, int64_t T, const cc_view* kring, const cc_view* vring, int32_t qk_norm, const cc_view* q_w, const cc_view* k_w, float eps,
                           const cc_view* freq, int32_t pairing, int32_t offset, float mag, int64_t pos0, int32_t H, int32_t G, int32_t dk, int32_t dv) {
    SEQ_F32(dev, kring, "qk_prepare_append kring"); SEQ_F32(dev, vring, "qk_prepare_append vring");
    CC_REQUIRE(dev, kring->ndim == 2 && pos0 >= 0 && qk_norm >= CC_QK_NORM_NONE && qk_norm <= CC_QK_NORM_ROW, "qk_prepare_append: bad arguments");
    const int64_t ring = kring->shape[0];
    CC_REQUIRE(dev, view_len(kring) == ring * G * dk && view_len(vring) == ring * G * dv, "qk_prepare_append: the rings do not fit kv=%d dk=%d dv=%d", G, dk, dv);
    CC_REQUIRE(dev, T <= ring, "qk_prepare_append: %lld tokens do not fit a ring of %lld", (long long)T, (long long)ring);
    const int64_t wq = qk_norm == CC_QK_NORM_ROW ? (int64_t)H * dk : dk, wk = qk_norm == CC_QK_NORM_ROW ? (int64_t)G * dk : dk;
    if (q_w) { SEQ_F32(dev, q_w, "qk_prepare_append q_w"); CC_REQUIRE(dev, qk_norm != CC_QK_NORM_NONE && view_len(q_w) == wq, "qk_prepare_append: q_w must have %lld elements", (long long)wq); }
    if (k_w) { SEQ_F32(dev, k_w, "qk_prepare_append k_w"); CC_REQUIRE(dev, qk_norm != CC_QK_NORM_NONE && view_len(k_w) == wk, "qk_prepare_append: k_w must have %lld elements", (long long)wk); }
    int64_t half = 0;
    if (freq) {
        SEQ_F32(dev, freq, "qk_prepare_append freq");
        half = view_len(freq);
        CC_REQUIRE(dev, offset >= 0 && offset + 2 * half <= dk && (pairing == CC_ROPE_NEIGHBOURS || pairing == CC_ROPE_HALVES), "qk_prepare_append: %lld pairs at column %d do not fit heads of %d",
                   (long long)half, offset, dk);
    }
    if (T == 0) return CC_OK;
    a.kring = fptr(kring); a.vring = fptr(vring); a.qw = q_w ? fptr(q_w) : nullptr; a.kw = k_w ? fptr(k_w) : nullptr;
    a.freq = freq ? fptr(freq) : nullptr; a.H = H; a.G = G; a.dk = dk; a.dv = dv; a.ring = (int)ring; a.norm = qk_norm; a.half = (int)half; a.off = offset;
    a.step = pairing == CC_ROPE_HALVES ? 1 : 2; a.gap = pairing == CC_ROPE_HALVES ? (int)half : 1; a.eps = eps; a.mag = mag; a.pos0 = pos0;
    CC_REQUIRE(dev, (H + G + 8) * 4 <= 48 * 1024, "qk_prepare_append: too many heads");
    const int blocks = qk_norm == CC_QK_NORM_ROW ? 1 : (H + G + QKP_THREADS / 32 - 1) / (QKP_THREADS / 32);       // a warp per head
    cc_launch_pdl(dev, qk_prepare_kernel, dim3((unsigned)T, (unsigned)blocks), QKP_THREADS, 0, a);
    CC_LAUNCH_CHECK(dev);
    return CC_OK;
}
extern "C" CC_API int cc_qk_prepare_append_cols(cc_device* dev, const cc_view* src, int32_t q_col0, int32_t k_col0, int32_t v_col0, const cc_view* kring, const cc_view* vring,
                                                int32_t qk_norm, const cc_view* q_w, const cc_view* k_w, float eps, const cc_view* freq, int32_t pairing, int32_t offset, float mag,
                                                int64_t pos0, int32_t H, int32_t G, int32_t dk, int32_t dv, cc_buf** out) {
    SEQ_ENTER(dev, "qk_prepare_append_cols");
    if (!out) return cc_fail(dev, CC_ERR_ARG, "qk_prepare_append_cols: out is NULL");
    SEQ_ROWS(dev, src, "qk_prepare_append_cols src");
    CC_REQUIRE(dev, H > 0 && G > 0 && dk > 0 && dv > 0, "qk_prepare_append_cols: bad arguments");
    const int64_t T = src->shape[0], cols = src->shape[1];
    CC_REQUIRE(dev, q_col0 >= 0 && k_col0 >= 0 && v_col0 >= 0 && q_col0 + (int64_t)H * dk <= cols && k_col0 + (int64_t)G * dk <= cols && v_col0 + (int64_t)G * dv <= cols,
               "qk_prepare_append_cols: columns %d / %d / %d of %lld do not fit heads=%d kv=%d dk=%d dv=%d", q_col0, k_col0, v_col0, (long long)cols, H, G, dk, dv);
    cc_buf* o = nullptr;
    int rc = cc_new_activation(dev, T * H * dk, CC_F32, false, &o);
    if (rc) return rc;
    QkPrepArgs a{};
    a.q = fptr(src) + q_col0; a.k = fptr(src) + k_col0; a.v = fptr(src) + v_col0; a.qo = (float*)o->base; a.qrs = a.krs = a.vrs = src->strides[0];
    rc = qk_prepare_impl(dev, a, T, kring, vring, qk_norm, q_w, k_w, eps, freq, pairing, offset, mag, pos0, H, G, dk, dv);
    if (rc) { cc_tensor_release(o); return rc; }
    *out = o;
    return CC_OK;
}
extern "C" CC_API int cc_qk_prepare_append(cc_device* dev, const cc_view* q, const cc_view* k, const cc_view* v, const cc_view* kring, const cc_view* vring, int32_t qk_norm,
                                           const cc_view* q_w, const cc_view* k_w, float eps, const cc_view* freq, int32_t pairing, int32_t offset, float mag, int64_t pos0,
                                           int32_t H, int32_t G, int32_t dk, int32_t dv) {
    SEQ_ENTER(dev, "qk_prepare_append");
    SEQ_F32(dev, q, "qk_prepare_append q"); SEQ_F32(dev, k, "qk_prepare_append k"); SEQ_F32(dev, v, "qk_prepare_append v");
    CC_REQUIRE(dev, H > 0 && G > 0 && dk > 0 && dv > 0 && q->ndim == 2, "qk_prepare_append: bad arguments");
    const int64_t T = q->shape[0];
    CC_REQUIRE(dev, view_len(q) == T * H * dk && view_len(k) == T * G * dk && view_len(v) == T * G * dv, "qk_prepare_append: operand sizes do not fit heads=%d kv=%d dk=%d dv=%d", H, G, dk, dv);
    QkPrepArgs a{};
    a.q = fptr(q); a.k = fptr(k); a.v = fptr(v); a.qo = fptr(q); a.qrs = (int64_t)H * dk; a.krs = (int64_t)G * dk; a.vrs = (int64_t)G * dv;
    return qk_prepare_impl(dev, a, T, kring, vring, qk_norm, q_w, k_w, eps, freq, pairing, offset, mag, pos0, H, G, dk, dv);
}

// ---- latent key/value cache ------------------------------------------------------------------------------------------------------------------
// one warp per token: the first `rank` columns are RMS-normalised and weighted, the pairs of the next columns rotated, the rest copied
struct LatAppend {
    float* ring;                  // NULL: nothing to append
    const float *ckv, *nw, *freq; // row t of the raw rows at ckv + t * rs
    int64_t rs, pos0;
    int ring_rows, rank, rest, half, step, gap;      // pair i of the rotated part: its columns step * i and step * i + gap
    float eps, mag;
};
#define LA_KEEP 16
__device__ __forceinline__ void latent_append_row(const LatAppend& a, int t, int lane) {
    const int rank = a.rank, cols = a.rank + a.rest, half = a.half;
    const int64_t pos0 = a.pos0;
    const float *nw = a.nw, *freq = a.freq, *src = a.ckv + t * a.rs;
    const float eps = a.eps, mag = a.mag;
    float* dst = a.ring + ((pos0 + t) % a.ring_rows) * cols;
    // the first 512 columns and their weights at once
    float keep[LA_KEEP], wt[LA_KEEP], ss = 0.0f;
#pragma unroll
    for (int e = 0; e < LA_KEEP; e++) {
        const int c = lane + e * 32;
        keep[e] = c < rank ? src[c] : 0.0f;
        wt[e] = nw && c < rank ? nw[c] : 1.0f;
    }
#pragma unroll
    for (int e = 0; e < LA_KEEP; e++) ss = fmaf(keep[e], keep[e], ss);
#pragma unroll 8
    for (int c = lane + LA_KEEP * 32; c < rank; c += 32) ss = fmaf(src[c], src[c], ss);
    ss = warp_sum(ss);
    const float inv = 1.0f / sqrtf(ss / (float)rank + eps);
#pragma unroll
    for (int e = 0; e < LA_KEEP; e++)
        if (lane + e * 32 < rank) dst[lane + e * 32] = keep[e] * inv * wt[e];
#pragma unroll 8
    for (int c = lane + LA_KEEP * 32; c < rank; c += 32) dst[c] = src[c] * inv * (nw ? nw[c] : 1.0f);
    for (int i = lane; i < half; i += 32) {
        float ou, ov;
        const int c = rank + a.step * i;
        rotate_pair(src[c], src[c + a.gap], (float)(pos0 + t), freq[i], mag, ou, ov);
        dst[c] = ou; dst[c + a.gap] = ov;
    }
    for (int c = rank + 2 * half + lane; c < cols; c += 32) dst[c] = src[c];
}
__global__ void latent_ring_append_kernel(LatAppend a, int T) {
    pdl_enter();
    const int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (t < T) latent_append_row(a, t, threadIdx.x & 31);
}
extern "C" CC_API int cc_latent_ring_append(cc_device* dev, const cc_view* ring, const cc_view* ckv, const cc_view* norm_w, float eps, int32_t rank, const cc_view* freq,
                                            float mag, int64_t pos0) {
    SEQ_ENTER(dev, "latent_ring_append");
    SEQ_F32(dev, ring, "latent_ring_append ring"); SEQ_F32(dev, ckv, "latent_ring_append ckv");
    if (norm_w) SEQ_F32(dev, norm_w, "latent_ring_append norm_w");
    if (freq) SEQ_F32(dev, freq, "latent_ring_append freq");
    CC_REQUIRE(dev, ring->ndim == 2 && ckv->ndim == 2 && ring->shape[1] == ckv->shape[1] && pos0 >= 0, "latent_ring_append: ring and rows must be 2-D with equal columns");
    const int64_t cols = ckv->shape[1], T = ckv->shape[0], half = freq ? view_len(freq) : 0;
    CC_REQUIRE(dev, rank >= 1 && rank + 2 * half <= cols && (!norm_w || view_len(norm_w) == rank), "latent_ring_append: rank %d + %lld rotated pairs do not fit %lld columns", rank,
               (long long)half, (long long)cols);
    CC_REQUIRE(dev, T <= ring->shape[0], "latent_ring_append: %lld tokens do not fit a ring of %lld", (long long)T, (long long)ring->shape[0]);
    if (T == 0) return CC_OK;
    const LatAppend a = {fptr(ring), fptr(ckv), norm_w ? fptr(norm_w) : nullptr, freq ? fptr(freq) : nullptr, cols, pos0, (int)ring->shape[0], rank, (int)(cols - rank), (int)half, 2, 1, eps, mag};
    cc_launch_pdl(dev, latent_ring_append_kernel, (unsigned)((T + 7) / 8), 256, 0, a, (int)T);
    CC_LAUNCH_CHECK(dev);
    return CC_OK;
}

// ---- per-head products: the up-projections of a latent cache, folded into the query and applied to the attention result ---------------------
struct HpArgs {
    const float *x, *W;           // token t's row at x + t * xrs, head h's inputs at + h * (n_in + rest)
    float* out;
    int64_t xrs, grs, pos0;
    const float *freq, *gate;     // gate (rest == 0 only): output (t, h, v) is multiplied by sigmoid(gate[t * grs + h * ghs + v * gvs]); NULL: not gated
    int T, H, n_in, rest, n_out, half, step, gap, ghs, gvs;
    float mag;
    LatAppend app;                // app.ring != NULL: the grid has one more z plane, the first, whose CTAs of head 0 write the tokens' cache rows
};
// grid (ceil(T / TOK), H, ceil(n_out / (8 * ROWS))): a warp owns ROWS neighbouring outputs of TOK tokens; its lanes read 4 columns each of W's rows (VEC) or one, the
// rows' pieces all at once, and the tokens' x from the cache: partial sums of every lane, then the butterfly -- one order per output, which n_in alone decides,
// whatever T is.  W: [H * n_out, n_in].  The `rest` columns behind a head's n_in inputs are copied behind its n_out outputs.
// Bound by latency: one token's 2 MB of W in 1024 warps, each with 4 loads of 16 bytes a lane in flight.  With 8 tokens staged in shared memory, whatever T was (32 turns of
// an integer division for 512 inputs), and 4-byte loads, 8 heads x 128 outputs of 512 took 15.8 us in a decoded token, x 512 outputs of 128 6.9 us; now 3.1 each.
#define HP_WARPS 8
template <int TOK, int ROWS, bool VEC>
__global__ void __launch_bounds__(HP_WARPS * 32) head_project_kernel(HpArgs a) {
    const int t0 = blockIdx.x * TOK, h = blockIdx.y, T = a.T, H = a.H, n_in = a.n_in, rest = a.rest, n_out = a.n_out, half = a.half;
    const int z = (int)blockIdx.z - (a.app.ring ? 1 : 0), lane = threadIdx.x & 31, v0 = (z * HP_WARPS + (threadIdx.x >> 5)) * ROWS;
    const int xs = n_in + rest, os = n_out + rest, nv = min(ROWS, n_out - v0);
    const float* W = a.W + ((int64_t)h * n_out + v0) * n_in;
    // the rows start for L2 while the kernel before is still at work
    if (z >= 0 && nv > 0)
        for (int64_t c = lane * 32; c < (int64_t)nv * n_in; c += 1024) asm volatile("prefetch.global.L2 [%0];" ::"l"(W + c));
    pdl_enter();
    if (z < 0) {
        if (h == 0)
            for (int tt = threadIdx.x >> 5; tt < TOK && t0 + tt < T; tt += HP_WARPS) latent_append_row(a.app, t0 + tt, lane);
        return;
    }
    const float* x = a.x + (int64_t)t0 * a.xrs + (int64_t)h * xs;
    const int nt = min(TOK, T - t0);
    if (nv > 0) {
        float acc[TOK][ROWS];
#pragma unroll
        for (int tt = 0; tt < TOK; tt++)
#pragma unroll
            for (int r = 0; r < ROWS; r++) acc[tt][r] = 0.0f;
        if (VEC) {
            const bool xvec = (((uintptr_t)x & 15) | (unsigned)(a.xrs & 3)) == 0;
#pragma unroll 4
            for (int d = lane * 4; d < n_in; d += 128) {
                float4 wv[ROWS];
#pragma unroll
                for (int r = 0; r < ROWS; r++) wv[r] = __ldg((const float4*)(W + (int64_t)min(r, nv - 1) * n_in + d));
#pragma unroll
                for (int tt = 0; tt < TOK; tt++) {
                    const float* xt = x + (int64_t)min(tt, nt - 1) * a.xrs + d;
                    const float4 xv = xvec ? *(const float4*)xt : make_float4(xt[0], xt[1], xt[2], xt[3]);
#pragma unroll
                    for (int r = 0; r < ROWS; r++) {
                        float y = acc[tt][r];
                        y = fmaf(xv.x, wv[r].x, y); y = fmaf(xv.y, wv[r].y, y); y = fmaf(xv.z, wv[r].z, y); y = fmaf(xv.w, wv[r].w, y);
                        acc[tt][r] = y;
                    }
                }
            }
        } else {
            for (int d = lane; d < n_in; d += 32)
#pragma unroll
                for (int r = 0; r < ROWS; r++) {
                    const float wv = W[(int64_t)min(r, nv - 1) * n_in + d];
#pragma unroll
                    for (int tt = 0; tt < TOK; tt++) acc[tt][r] = fmaf(x[(int64_t)min(tt, nt - 1) * a.xrs + d], wv, acc[tt][r]);
                }
        }
#pragma unroll
        for (int tt = 0; tt < TOK; tt++)
#pragma unroll
            for (int r = 0; r < ROWS; r++) {
                float sum = warp_sum(acc[tt][r]);
                if (lane != 0 || tt >= nt || r >= nv) continue;
                if (a.gate) sum *= seq_sigmoid(a.gate[(t0 + tt) * a.grs + h * a.ghs + (v0 + r) * a.gvs]);
                a.out[((int64_t)(t0 + tt) * H + h) * os + v0 + r] = sum;
            }
    }
    if (z == 0 && rest > 0) {
        // the carried columns: the first 2 * half of them are rotated on the way when a frequency table is given
        for (int tt = 0; tt < nt; tt++) {
            const float* src = x + tt * a.xrs + n_in;
            float* dst = a.out + ((int64_t)(t0 + tt) * H + h) * os + n_out;
            for (int p = threadIdx.x; p < half; p += HP_WARPS * 32)
                rotate_pair(src[a.step * p], src[a.step * p + a.gap], (float)(a.pos0 + t0 + tt), a.freq[p], a.mag, dst[a.step * p], dst[a.step * p + a.gap]);
            for (int j = 2 * half + threadIdx.x; j < rest; j += HP_WARPS * 32) dst[j] = src[j];
        }
    }
}
template <int TOK, int ROWS, bool VEC>
static int head_project_launch(cc_device* dev, const HpArgs& a) {
    cc_launch_pdl(dev, head_project_kernel<TOK, ROWS, VEC>, dim3((unsigned)((a.T + TOK - 1) / TOK), (unsigned)a.H, (unsigned)((a.n_out + HP_WARPS * ROWS - 1) / (HP_WARPS * ROWS) + (a.app.ring ? 1 : 0))),
                  HP_WARPS * 32, 0, a);
    CC_LAUNCH_CHECK(dev);
    return CC_OK;
}
static int head_project_few(cc_device* dev, const HpArgs& a) {
    CC_REQUIRE(dev, (int64_t)8 * a.n_in * 4 <= 160 * 1024, "head_project: %d inputs per head are too many", a.n_in);
    if (a.n_in & 3 || (uintptr_t)a.W & 15) return head_project_launch<4, 1, false>(dev, a);
    // rows of fewer than 256 columns by fours: a lane's one or two pieces of a row are too little in flight
    if (a.n_in < 256) return a.T == 1 ? head_project_launch<1, 4, true>(dev, a) : head_project_launch<4, 4, true>(dev, a);
    return a.T == 1 ? head_project_launch<1, 1, true>(dev, a) : head_project_launch<4, 2, true>(dev, a);
}
// many rows and nothing carried: a 64 x 64 output tile of one head per CTA, 16-deep slices of the inputs through shared memory, 4 x 4 outputs
// per thread, every sum over n_in in ascending order inside one thread.  grid (ceil(n_out / 64), ceil(T / 64), H)
#define HPT_TILE 64
#define HPT_K 16
__global__ void __launch_bounds__(256) head_project_tile_kernel(const float* __restrict__ x, const float* __restrict__ W, float* __restrict__ out, int T, int H, int n_in, int n_out) {
    pdl_enter();
    __shared__ float sw[HPT_K][HPT_TILE + 4];
    __shared__ float sx[HPT_K][HPT_TILE + 4];
    const int o0 = blockIdx.x * HPT_TILE, t0 = blockIdx.y * HPT_TILE, h = blockIdx.z;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const float* Wh = W + (int64_t)h * n_out * n_in;
    const int64_t xrs = (int64_t)H * n_in, ors = (int64_t)H * n_out;
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = 0.0f;
    for (int k0 = 0; k0 < n_in; k0 += HPT_K) {
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const int idx = threadIdx.x + e * 256;
            const int r = idx >> 4, kk = idx & 15;
            const bool kin = k0 + kk < n_in;
            sw[kk][r] = (kin && o0 + r < n_out) ? Wh[(int64_t)(o0 + r) * n_in + k0 + kk] : 0.0f;
            sx[kk][r] = (kin && t0 + r < T) ? x[(int64_t)(t0 + r) * xrs + h * n_in + k0 + kk] : 0.0f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < HPT_K; kk++) {
            const float4 wv = *(const float4*)&sw[kk][tx * 4];
            const float4 xv = *(const float4*)&sx[kk][ty * 4];
            const float wr[4] = {wv.x, wv.y, wv.z, wv.w}, xr[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = fmaf(xr[i], wr[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int t = t0 + ty * 4 + i;
        if (t >= T) continue;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int o = o0 + tx * 4 + j;
            if (o < n_out) out[(int64_t)t * ors + h * n_out + o] = acc[i][j];
        }
    }
}
extern "C" CC_API int cc_head_project(cc_device* dev, const cc_view* x, const cc_view* w, int32_t n_heads, int32_t rest, const cc_view* freq, float mag, int64_t pos0,
                                      cc_buf** out) {
    SEQ_ENTER(dev, "head_project");
    if (freq) { SEQ_F32(dev, freq, "head_project freq"); CC_REQUIRE(dev, 2 * view_len(freq) <= rest && pos0 >= 0, "head_project: more rotated pairs than carried columns"); }
    if (!out) return cc_fail(dev, CC_ERR_ARG, "head_project: out is NULL");
    SEQ_F32(dev, x, "head_project x"); SEQ_F32(dev, w, "head_project w");
    CC_REQUIRE(dev, x->ndim == 2 && w->ndim == 2 && n_heads > 0 && rest >= 0 && w->shape[0] % n_heads == 0 && x->shape[1] == (int64_t)n_heads * (w->shape[1] + rest),
               "head_project: x must be [T, heads * (n_in + rest)] and w [heads * n_out, n_in]");
    const int64_t T = x->shape[0], n_in = w->shape[1], n_out = w->shape[0] / n_heads;
    CC_REQUIRE(dev, n_in * 32 <= 160 * 1024, "head_project: %lld inputs per head are too many", (long long)n_in);
    cc_buf* o = nullptr;
    int rc = cc_new_activation(dev, T * n_heads * (n_out + rest), CC_F32, false, &o);
    if (rc) return rc;
    *out = o;
    if (T == 0) return CC_OK;
    if (rest == 0 && T >= 64) {          // a pass of many rows (a prompt): tiles; the sums differ from the few-row kernel's by their order only
        cc_launch_pdl(dev, head_project_tile_kernel, dim3((unsigned)((n_out + HPT_TILE - 1) / HPT_TILE), (unsigned)((T + HPT_TILE - 1) / HPT_TILE), (unsigned)n_heads), 256, 0, fptr(x), fptr(w), (float*)o->base, (int)T, n_heads, (int)n_in, (int)n_out);
        CC_LAUNCH_CHECK(dev);
        return CC_OK;
    }
    HpArgs a{};
    a.x = fptr(x); a.W = fptr(w); a.out = (float*)o->base; a.xrs = x->shape[1]; a.pos0 = pos0; a.freq = freq ? fptr(freq) : nullptr; a.half = freq ? (int)view_len(freq) : 0; a.mag = mag;
    a.T = (int)T; a.H = n_heads; a.n_in = (int)n_in; a.rest = rest; a.n_out = (int)n_out; a.step = 2; a.gap = 1;
    return head_project_few(dev, a);
}
static int head_project_gated_impl(cc_device* dev, const cc_view* x, const cc_view* w, int32_t n_heads, const cc_view* gate_src, int32_t gate_col0, bool per_head, cc_buf** out);
extern "C" CC_API int cc_head_project_gated(cc_device* dev, const cc_view* x, const cc_view* w, int32_t n_heads, const cc_view* gate_src, int32_t gate_col0, cc_buf** out) {
    return head_project_gated_impl(dev, x, w, n_heads, gate_src, gate_col0, false, out);
}
extern "C" CC_API int cc_head_project_head_gated(cc_device* dev, const cc_view* x, const cc_view* w, int32_t n_heads, const cc_view* gate_src, int32_t gate_col0, cc_buf** out) {
    return head_project_gated_impl(dev, x, w, n_heads, gate_src, gate_col0, true, out);
}
// per_head: one gate number per head instead of one per output column
static int head_project_gated_impl(cc_device* dev, const cc_view* x, const cc_view* w, int32_t n_heads, const cc_view* gate_src, int32_t gate_col0, bool per_head, cc_buf** out) {
    SEQ_ENTER(dev, "head_project_gated");
    if (!out) return cc_fail(dev, CC_ERR_ARG, "head_project_gated: out is NULL");
    SEQ_F32(dev, x, "head_project_gated x"); SEQ_F32(dev, w, "head_project_gated w"); SEQ_ROWS(dev, gate_src, "head_project_gated gate");
    CC_REQUIRE(dev, x->ndim == 2 && w->ndim == 2 && n_heads > 0 && w->shape[0] % n_heads == 0 && x->shape[1] == (int64_t)n_heads * w->shape[1],
               "head_project_gated: x must be [T, heads * n_in] and w [heads * n_out, n_in]");
    const int64_t T = x->shape[0];
    const int64_t gates = per_head ? n_heads : w->shape[0];
    CC_REQUIRE(dev, gate_src->shape[0] == T && gate_col0 >= 0 && gate_col0 + gates <= gate_src->shape[1], "head_project_gated: the gate needs %lld columns from column %d on",
               (long long)gates, gate_col0);
    cc_buf* o = nullptr;
    int rc = cc_new_activation(dev, T * w->shape[0], CC_F32, false, &o);
    if (rc) return rc;
    *out = o;
    if (T == 0) return CC_OK;
    HpArgs a{};
    a.x = fptr(x); a.W = fptr(w); a.out = (float*)o->base; a.xrs = x->shape[1]; a.gate = fptr(gate_src) + gate_col0; a.grs = gate_src->strides[0]; a.mag = 1.0f;
    a.T = (int)T; a.H = n_heads; a.n_in = (int)w->shape[1]; a.n_out = (int)(w->shape[0] / n_heads);
    a.ghs = per_head ? 1 : a.n_out; a.gvs = per_head ? 0 : 1;
    return head_project_few(dev, a);
}
extern "C" CC_API int cc_latent_query_append(cc_device* dev, const cc_view* q_src, int32_t q_col0, const cc_view* uk_t, int32_t n_heads, int32_t rest, const cc_view* freq, float mag,
                                             int64_t pos0, const cc_view* kv_src, int32_t kv_col0, const cc_view* ring, const cc_view* norm_w, float eps, cc_buf** out) {
    return cc_latent_query_append_paired(dev, q_src, q_col0, uk_t, n_heads, rest, freq, CC_ROPE_NEIGHBOURS, mag, pos0, kv_src, kv_col0, ring, norm_w, eps, out);
}
extern "C" CC_API int cc_latent_query_append_paired(cc_device* dev, const cc_view* q_src, int32_t q_col0, const cc_view* uk_t, int32_t n_heads, int32_t rest, const cc_view* freq,
                                                    int32_t pairing, float mag, int64_t pos0, const cc_view* kv_src, int32_t kv_col0, const cc_view* ring, const cc_view* norm_w,
                                                    float eps, cc_buf** out) {
    SEQ_ENTER(dev, "latent_query_append");
    CC_REQUIRE(dev, pairing == CC_ROPE_NEIGHBOURS || pairing == CC_ROPE_HALVES, "latent_query_append: unknown pairing %d", pairing);
    if (!out) return cc_fail(dev, CC_ERR_ARG, "latent_query_append: out is NULL");
    SEQ_ROWS(dev, q_src, "latent_query_append q"); SEQ_F32(dev, uk_t, "latent_query_append uk_t");
    CC_REQUIRE(dev, uk_t->ndim == 2 && n_heads > 0 && rest >= 0 && uk_t->shape[0] % n_heads == 0 && pos0 >= 0, "latent_query_append: bad arguments");
    const int64_t T = q_src->shape[0], dim = uk_t->shape[1], rank = uk_t->shape[0] / n_heads;
    CC_REQUIRE(dev, q_col0 >= 0 && q_col0 + n_heads * (dim + rest) <= q_src->shape[1], "latent_query_append: the queries need %lld columns from column %d on",
               (long long)(n_heads * (dim + rest)), q_col0);
    if (freq) { SEQ_F32(dev, freq, "latent_query_append freq"); CC_REQUIRE(dev, 2 * view_len(freq) <= rest, "latent_query_append: more rotated pairs than carried columns"); }
    HpArgs a{};
    const int half = freq ? (int)view_len(freq) : 0, step = pairing == CC_ROPE_HALVES ? 1 : 2, gap = pairing == CC_ROPE_HALVES ? half : 1;
    if (kv_src) {
        SEQ_ROWS(dev, kv_src, "latent_query_append kv"); SEQ_F32(dev, ring, "latent_query_append ring");
        if (norm_w) { SEQ_F32(dev, norm_w, "latent_query_append norm_w"); CC_REQUIRE(dev, view_len(norm_w) == rank, "latent_query_append: norm_w must have %lld elements", (long long)rank); }
        CC_REQUIRE(dev, ring->ndim == 2 && ring->shape[1] == rank + rest && T <= ring->shape[0] && kv_src->shape[0] == T && kv_col0 >= 0 && kv_col0 + rank + rest <= kv_src->shape[1],
                   "latent_query_append: ring rows have rank + rest columns and so have the raw rows from column %d on", kv_col0);
        a.app = {fptr(ring), fptr(kv_src) + kv_col0, norm_w ? fptr(norm_w) : nullptr, freq ? fptr(freq) : nullptr, kv_src->strides[0], pos0, (int)ring->shape[0], (int)rank, rest,
                 half, step, gap, eps, mag};
    }
    cc_buf* o = nullptr;
    int rc = cc_new_activation(dev, T * n_heads * (rank + rest), CC_F32, false, &o);
    if (rc) return rc;
    *out = o;
    if (T == 0) return CC_OK;
    a.x = fptr(q_src) + q_col0; a.W = fptr(uk_t); a.out = (float*)o->base; a.xrs = q_src->strides[0]; a.pos0 = pos0; a.freq = freq ? fptr(freq) : nullptr;
    a.half = half; a.step = step; a.gap = gap; a.mag = mag; a.T = (int)T; a.H = n_heads; a.n_in = (int)dim; a.rest = rest; a.n_out = (int)rank;
    return head_project_few(dev, a);
}
// the same for a pass of many rows, whose queries are not folded: one CTA per token copies the queries out of their columns, a warp a head, rotating the last
// `rest` columns on the way (a pair by the lane of its first column), and one more warp writes the token's cache row.  512 rows of 8 heads (128 + 64), cache rows of
// 512 + 64, us: elements dealt to threads by a division, the cache row behind them 5.5 ; here 3.6
#define LP_WARPS 8
__global__ void __launch_bounds__(LP_WARPS * 32 + 32) latent_prepare_kernel(const float* __restrict__ q, int64_t qrs, float* __restrict__ out, int H, int dim, LatAppend a) {
    pdl_enter();
    const int t = blockIdx.x, hs = dim + a.rest, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (w == LP_WARPS) {
        if (a.ring) latent_append_row(a, t, lane);
        return;
    }
    for (int h = w; h < H; h += LP_WARPS) {
        const float* src = q + t * qrs + (int64_t)h * hs;
        float* dst = out + ((int64_t)t * H + h) * hs;
        for (int i = lane; i < a.half; i += 32) {
            float ou, ov;
            const int c = dim + a.step * i;
            rotate_pair(src[c], src[c + a.gap], (float)(a.pos0 + t), a.freq[i], a.mag, ou, ov);
            dst[c] = ou; dst[c + a.gap] = ov;
        }
#pragma unroll 4
        for (int c = lane; c < dim; c += 32) dst[c] = src[c];
        for (int c = dim + 2 * a.half + lane; c < hs; c += 32) dst[c] = src[c];
    }
}
extern "C" CC_API int cc_latent_prepare_append(cc_device* dev, const cc_view* q_src, int32_t q_col0, int32_t n_heads, int32_t dim, int32_t rest, const cc_view* freq, int32_t pairing,
                                               float mag, int64_t pos0, const cc_view* kv_src, int32_t kv_col0, const cc_view* ring, const cc_view* norm_w, float eps, cc_buf** out) {
    SEQ_ENTER(dev, "latent_prepare_append");
    if (!out) return cc_fail(dev, CC_ERR_ARG, "latent_prepare_append: out is NULL");
    SEQ_ROWS(dev, q_src, "latent_prepare_append q");
    CC_REQUIRE(dev, n_heads > 0 && dim > 0 && rest >= 0 && pos0 >= 0 && (pairing == CC_ROPE_NEIGHBOURS || pairing == CC_ROPE_HALVES), "latent_prepare_append: bad arguments");
    const int64_t T = q_src->shape[0], cols = (int64_t)n_heads * (dim + rest);
    CC_REQUIRE(dev, q_col0 >= 0 && q_col0 + cols <= q_src->shape[1], "latent_prepare_append: the queries need %lld columns from column %d on", (long long)cols, q_col0);
    if (freq) { SEQ_F32(dev, freq, "latent_prepare_append freq"); CC_REQUIRE(dev, 2 * view_len(freq) <= rest, "latent_prepare_append: more rotated pairs than rotated columns"); }
    LatAppend a{};
    a.freq = freq ? fptr(freq) : nullptr; a.half = freq ? (int)view_len(freq) : 0; a.step = pairing == CC_ROPE_HALVES ? 1 : 2; a.gap = pairing == CC_ROPE_HALVES ? a.half : 1;
    a.rest = rest; a.eps = eps; a.mag = mag; a.pos0 = pos0;
    if (kv_src) {
        SEQ_ROWS(dev, kv_src, "latent_prepare_append kv"); SEQ_F32(dev, ring, "latent_prepare_append ring");
        CC_REQUIRE(dev, ring->ndim == 2 && ring->shape[1] > rest && T <= ring->shape[0] && kv_src->shape[0] == T && kv_col0 >= 0 && kv_col0 + ring->shape[1] <= kv_src->shape[1],
                   "latent_prepare_append: the raw rows need a ring row's columns from column %d on", kv_col0);
        a.rank = (int)(ring->shape[1] - rest);
        if (norm_w) { SEQ_F32(dev, norm_w, "latent_prepare_append norm_w"); CC_REQUIRE(dev, view_len(norm_w) == a.rank, "latent_prepare_append: norm_w must have %d elements", a.rank); }
        a.ring = fptr(ring); a.ckv = fptr(kv_src) + kv_col0; a.nw = norm_w ? fptr(norm_w) : nullptr; a.rs = kv_src->strides[0]; a.ring_rows = (int)ring->shape[0];
    }
    cc_buf* o = nullptr;
    int rc = cc_new_activation(dev, T * cols, CC_F32, false, &o);
    if (rc) return rc;
    *out = o;
    if (T == 0) return CC_OK;
    cc_launch_pdl(dev, latent_prepare_kernel, (unsigned)T, LP_WARPS * 32 + 32, 0, fptr(q_src) + q_col0, q_src->strides[0], (float*)o->base, n_heads, dim, a);
    CC_LAUNCH_CHECK(dev);
    return CC_OK;
}

// out[j, h] = [ a[j, h, :dim] | shared[j, col0 : col0 + rest] ]: every head's part followed by the columns all heads share.  One thread per element.
__global__ void head_concat_shared_kernel(const float* __restrict__ a, const float* __restrict__ shared, float* __restrict__ out, int64_t n, int H, int dim, int rest, int scols,
                                          int col0) {
    pdl_enter();
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= n) return;
    const int hs = dim + rest;
    const int c = (int)(idx % hs);
    const int64_t jh = idx / hs, j = jh / H;
    out[idx] = c < dim ? a[jh * dim + c] : shared[j * scols + col0 + (c - dim)];
}
// the same, four neighbouring columns per thread: grid (columns of a row / 512, rows).  2048 rows of 8 x (128 + 64), us: one element by 64-bit divisions 14.1 ; here 6.9
__global__ void __launch_bounds__(128) head_concat_shared4_kernel(const float* __restrict__ a, const float* __restrict__ shared, float* __restrict__ out, int H, int dim, int rest, int scols, int col0) {
    pdl_enter();
    const int hs = dim + rest, at = (blockIdx.x * 128 + threadIdx.x) * 4;
    if (at >= H * hs) return;
    const int h = at / hs, c = at - h * hs;
    const int64_t j = blockIdx.y;
    *(float4*)(out + j * H * hs + at) = c < dim ? *(const float4*)(a + (j * H + h) * dim + c) : *(const float4*)(shared + j * scols + col0 + (c - dim));
}
extern "C" CC_API int cc_head_concat_shared(cc_device* dev, const cc_view* a, const cc_view* shared, int32_t n_heads, int32_t col0, int32_t rest, cc_buf** out) {
    SEQ_ENTER(dev, "head_concat_shared");
    if (!out) return cc_fail(dev, CC_ERR_ARG, "head_concat_shared: out is NULL");
    SEQ_F32(dev, a, "head_concat_shared a"); SEQ_F32(dev, shared, "head_concat_shared shared");
    CC_REQUIRE(dev, a->ndim == 2 && shared->ndim == 2 && n_heads > 0 && a->shape[1] % n_heads == 0 && shared->shape[0] >= a->shape[0] && col0 >= 0 && rest >= 0 &&
                        col0 + rest <= shared->shape[1],
               "head_concat_shared: a must be [rows, heads * dim], shared [>= rows, cols] with cols >= col0 + rest");
    const int64_t rows = a->shape[0], dim = a->shape[1] / n_heads;
    cc_buf* o = nullptr;
    int rc = cc_new_activation(dev, rows * n_heads * (dim + rest), CC_F32, false, &o);
    if (rc) return rc;
    *out = o;
    const int64_t n = rows * n_heads * (dim + rest);
    if (n == 0) return CC_OK;
    const int scols = (int)shared->shape[1];
    if (dim % 4 == 0 && rest % 4 == 0 && scols % 4 == 0 && col0 % 4 == 0 && rows <= 65535 && (((uintptr_t)fptr(a) | (uintptr_t)fptr(shared)) & 15) == 0)
        cc_launch_pdl(dev, head_concat_shared4_kernel, dim3((unsigned)((n_heads * (dim + rest) / 4 + 127) / 128), (unsigned)rows), 128, 0, fptr(a), fptr(shared), (float*)o->base, n_heads, (int)dim, rest, scols, col0);
    else cc_launch_pdl(dev, head_concat_shared_kernel, (unsigned)((n + 255) / 256), 256, 0, fptr(a), fptr(shared), (float*)o->base, n, n_heads, (int)dim, rest, scols, col0);
    CC_LAUNCH_CHECK(dev);
    return CC_OK;
}

// ---- column blocks of one product's result as separate tensors ------------------------------------------------------------------------------
#define SPLIT_MAX 16
struct SplitArgs {
    float* dst[SPLIT_MAX];
    int end[SPLIT_MAX];          // first column behind part p
    int n;
};
// grid (ceil(cols / 256), about rows / 8): a thread owns one column (its part is found once) and walks the rows of its grid line
__global__ void split_cols_kernel(const float* __restrict__ src, SplitArgs a, int64_t rows, int cols) {
    pdl_enter();
    const int c = blockIdx.x * 256 + threadIdx.x;
    if (c >= cols) return;
    int p = 0;
    while (p + 1 < a.n && c >= a.end[p]) p++;
    const int begin = p ? a.end[p - 1] : 0, w = a.end[p] - begin;
    float* dst = a.dst[p] + (c - begin);
    for (int64_t r = blockIdx.y; r < rows; r += gridDim.y) dst[r * w] = src[r * cols + c];
}
extern "C" CC_API int cc_split_cols(cc_device* dev, const cc_view* src, int32_t n_parts, const int32_t* widths, cc_buf** outs) {
    SEQ_ENTER(dev, "split_cols");
    if (!widths || !outs) return cc_fail(dev, CC_ERR_ARG, "split_cols: widths / outs is NULL");
    SEQ_F32(dev, src, "split_cols src");
    CC_REQUIRE(dev, src->ndim == 2 && n_parts >= 1 && n_parts <= SPLIT_MAX, "split_cols: src must be [rows, cols], 1..%d parts", SPLIT_MAX);
    const int64_t rows = src->shape[0], cols = src->shape[1];
    int64_t sum = 0;
    for (int p = 0; p < n_parts; p++) { CC_REQUIRE(dev, widths[p] >= 1, "split_cols: empty part %d", p); sum += widths[p]; }
    CC_REQUIRE(dev, sum == cols, "split_cols: the parts have %lld columns, src %lld", (long long)sum, (long long)cols);
    SplitArgs a;
    a.n = n_parts;
    int end = 0;
    for (int p = 0; p < n_parts; p++) {
        cc_buf* o = nullptr;
        int rc = cc_new_activation(dev, rows * widths[p], CC_F32, false, &o);
        if (rc) { for (int q = 0; q < p; q++) { cc_tensor_release(outs[q]); outs[q] = nullptr; } return rc; }
        outs[p] = o;
        a.dst[p] = (float*)o->base;
        a.end[p] = (end += widths[p]);
    }
    const int64_t total = rows * cols;
    if (total == 0) return CC_OK;
    const int64_t lines = (rows + 7) / 8;             // a thread copies about 8 rows of its column
    cc_launch_pdl(dev, split_cols_kernel, dim3((unsigned)((cols + 255) / 256), (unsigned)(lines < 65535 ? lines : 65535)), 256, 0, fptr(src), a, rows, (int)cols);
    CC_LAUNCH_CHECK(dev);
    return CC_OK;
}

// ---- PolyNorm ------------------------------------------------------------------------------------------------------------------------------
// one CTA per row: thread-strided sums of z^2, z^4, z^6, a fixed tree over the 256 partial sums, then the weighted sum of the three unit powers
__global__ void __launch_bounds__(256) poly_norm_kernel(float* __restrict__ z, const float* __restrict__ coef, int cols, float eps) {
    pdl_enter();
    __shared__ float red[3][8];
    float* zr = z + (int64_t)blockIdx.x * cols;
    float s2 = 0.0f, s4 = 0.0f, s6 = 0.0f;
    for (int c = threadIdx.x; c < cols; c += 256) {
        const float v = zr[c], v2 = v * v, v3 = v2 * v;
        s2 += v2; s4 = fmaf(v2, v2, s4); s6 = fmaf(v3, v3, s6);
    }
    s2 = warp_sum(s2); s4 = warp_sum(s4); s6 = warp_sum(s6);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) { red[0][warp] = s2; red[1][warp] = s4; red[2][warp] = s6; }
    __syncthreads();
    float t2 = 0.0f, t4 = 0.0f, t6 = 0.0f;
#pragma unroll
    for (int w = 0; w < 8; w++) { t2 += red[0][w]; t4 += red[1][w]; t6 += red[2][w]; }
    const float i1 = 1.0f / sqrtf(t2 / (float)cols + eps), i2 = 1.0f / sqrtf(t4 / (float)cols + eps), i3 = 1.0f / sqrtf(t6 / (float)cols + eps);
    const float a = coef[0], b = coef[1], c3 = coef[2], e = coef[3];
    for (int c = threadIdx.x; c < cols; c += 256) {
        const float v = zr[c], v2 = v * v, v3 = v2 * v;
        zr[c] = a * (v * i1) + b * (v2 * i2) + c3 * (v3 * i3) + e;
    }
}
extern "C" CC_API int cc_poly_norm(cc_device* dev, const cc_view* z, const cc_view* coef, float eps) {
    SEQ_ENTER(dev, "poly_norm");
    SEQ_F32(dev, z, "poly_norm z"); SEQ_F32(dev, coef, "poly_norm coef");
    CC_REQUIRE(dev, z->ndim == 2 && view_len(coef) == 4, "poly_norm: z must be [rows, cols] and coef hold 4 numbers");
    if (z->shape[0] == 0) return CC_OK;
    cc_launch_pdl(dev, poly_norm_kernel, (unsigned)z->shape[0], 256, 0, fptr(z), fptr(coef), (int)z->shape[1], eps);
    CC_LAUNCH_CHECK(dev);
    return CC_OK;
}

// ---- gated sum of sublayer results into the residual stream -----------------------------------------------------------------------------------
__global__ void gated_sum_kernel(float* __restrict__ dst, const float* __restrict__ y1, const float* __restrict__ g1, const float* __restrict__ b1, const float* __restrict__ y2,
                                 const float* __restrict__ g2, const float* __restrict__ b2, int64_t n, int cols, int accumulate) {
    pdl_enter();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int c = (int)(i % cols);
    float v = y1[i];
    if (g1) v *= seq_sigmoid(g1[i] + (b1 ? b1[c] : 0.0f));
    if (y2) {
        float u = y2[i];
        if (g2) u *= seq_sigmoid(g2[i] + (b2 ? b2[c] : 0.0f));
        v += u;
    }
    dst[i] = accumulate ? dst[i] + v : v;
}
extern "C" CC_API int cc_gated_sum(cc_device* dev, const cc_view* dst, int32_t accumulate, const cc_view* y1, const cc_view* g1, const cc_view* b1, const cc_view* y2,
                                   const cc_view* g2, const cc_view* b2) {
    SEQ_ENTER(dev, "gated_sum");
    SEQ_F32(dev, dst, "gated_sum dst"); SEQ_F32(dev, y1, "gated_sum y1");
    CC_REQUIRE(dev, dst->ndim == 2, "gated_sum: dst must be [rows, cols]");
    const int64_t n = view_len(dst), cols = dst->shape[1];
    const cc_view* same[] = {y1, g1, y2, g2};
    for (const cc_view* v : same)
        if (v) { SEQ_F32(dev, v, "gated_sum operand"); CC_REQUIRE(dev, view_len(v) == n, "gated_sum: an operand has %lld elements, dst %lld", (long long)view_len(v), (long long)n); }
    const cc_view* bias[] = {b1, b2};
    for (const cc_view* v : bias)
        if (v) { SEQ_F32(dev, v, "gated_sum bias"); CC_REQUIRE(dev, view_len(v) == cols, "gated_sum: a bias needs one number per column"); }
    CC_REQUIRE(dev, (!b1 || g1) && (!b2 || g2) && (!g2 || y2), "gated_sum: a bias needs its gate, a gate its operand");
    if (n == 0) return CC_OK;
    cc_launch_pdl(dev, gated_sum_kernel, (unsigned)((n + 255) / 256), 256, 0, fptr(dst), fptr(y1), g1 ? fptr(g1) : nullptr, b1 ? fptr(b1) : nullptr, y2 ? fptr(y2) : nullptr,
                                                                           g2 ? fptr(g2) : nullptr, b2 ? fptr(b2) : nullptr, n, (int)cols, accumulate);
    CC_LAUNCH_CHECK(dev);
    return CC_OK;
}
