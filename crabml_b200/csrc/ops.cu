// ops.cu -- the small ops around the matvec, one launch per trait call.
// Compiled with -fmad=false / IEEE div+sqrt so that every op reproduces the reference's f32
// arithmetic; only reduction ORDER differs (the canonical 512-thread tree of common.cuh instead of sequential).
#include "common.cuh"
#include "split_gemm.cuh"

// ---- rms_norm_inplace: primitives/rms_norm.rs:32-47  x /= sqrt(sum(x^2)/n + eps), no weight ------------
// canonical 512-thread order (common.cuh); cols % 4 == 0 is implied by the reference's own assert (cols % 32 == 0)
__global__ void __launch_bounds__(CC_RED_THREADS) rms_norm_kernel(float* x, int64_t cols, float eps) {
    pdl_enter();
    __shared__ float sh[CC_RED_WARPS];
    float* v = x + (int64_t)blockIdx.x * cols;
    float s = 0.0f;
    const int64_t n4 = cols >> 2;
    for (int64_t i = threadIdx.x; i < n4; i += CC_RED_THREADS) { const float* c = v + 4 * i; s += cc_sq4(make_float4(c[0], c[1], c[2], c[3])); }
    if ((cols & 3) && threadIdx.x == 0) for (int64_t i = n4 * 4; i < cols; i++) s += v[i] * v[i];
    s = cc_block_sum_512(s, sh);
    float rms = sqrtf(s / (float)cols + eps);
    for (int64_t i = threadIdx.x; i < cols; i += CC_RED_THREADS) v[i] = v[i] / rms;
}
int cc_launch_rms_norm(cc_device* dev, float* x, int64_t rows, int64_t cols, float eps) {
    if (rows == 0 || cols == 0) return CC_OK;
    cc_launch_pdl(dev, rms_norm_kernel, (unsigned)rows, CC_RED_THREADS, 0, x, cols, eps);
    CC_LAUNCH_CHECK(dev);
    return CC_OK;
}

// rope_inplace lives in exact.cu (host-evaluated cos/sin table, used by both modes)

// ---- softmax_inplace: primitives/softmax.rs:39-54 with the f16 exp LUT (quirk B4) ---------------------------
__device__ __forceinline__ float exp_cached(float v, const uint16_t* lut) { return h2f_bits(lut[f2h_bits(v)]); }

__global__ void __launch_bounds__(CC_RED_THREADS) softmax_kernel(float* x, int64_t cols, const uint16_t* __restrict__ lut) {
    pdl_enter();
    __shared__ float sh[CC_RED_WARPS];
    float* v = x + (int64_t)blockIdx.x * cols;
    float m = -INFINITY;
    for (int64_t i = threadIdx.x; i < cols; i += CC_RED_THREADS) m = fmaxf(m, v[i]);
    m = cc_block_max_512(m, sh);
    float s = 0.0f;
    for (int64_t i = threadIdx.x; i < cols; i += CC_RED_THREADS) {
        float e = exp_cached(v[i] - m, lut);
        v[i] = e;
        s += e;
    }
    s = cc_block_sum_512(s, sh);          // canonical order (common.cuh): same bits as the fused attention kernels
    for (int64_t i = threadIdx.x; i < cols; i += CC_RED_THREADS) v[i] = v[i] / s;
}
// many rows: a warp per row with the sums of softmax_kernel -- lane l of its w-th warp is here lane l's w-th partial sum, so the bits are the same -- and
// no barrier.  16384 rows of 512 (a prompt of 512 tokens, 32 heads): 74 -> 23 us, bound by the gathers from the 128 KB exponential table
#define SM_MAX_COLS 2048
#define SM_WARPS 4
__global__ void __launch_bounds__(SM_WARPS * 32) softmax_rows_kernel(float* x, int64_t rows, int cols, const uint16_t* __restrict__ lut) {
    pdl_enter();
    const int lane = threadIdx.x & 31;
    const int64_t row = (int64_t)blockIdx.x * SM_WARPS + (threadIdx.x >> 5);
    if (row >= rows) return;
    float* v = x + row * cols;
    float m = -INFINITY, part[CC_RED_WARPS];
#pragma unroll 4
    for (int i = lane; i < cols; i += 32) m = fmaxf(m, v[i]);
    m = warp_max(m);
#pragma unroll
    for (int w = 0; w < CC_RED_WARPS; w++) part[w] = 0.0f;
    for (int c0 = 0; c0 < cols; c0 += CC_RED_THREADS) {
#pragma unroll
        for (int w = 0; w < CC_RED_WARPS; w++) {
            const int i = c0 + 32 * w + lane;
            if (i < cols) {
                const float e = exp_cached(v[i] - m, lut);
                v[i] = e;
                part[w] += e;
            }
        }
    }
    float s = 0.0f;
#pragma unroll
    for (int w = 0; w < CC_RED_WARPS; w++) s += warp_sum(part[w]);
#pragma unroll 4
    for (int i = lane; i < cols; i += 32) v[i] = v[i] / s;
}
int cc_launch_softmax(cc_device* dev, float* x, int64_t rows, int64_t cols) {
    if (rows == 0 || cols == 0) return CC_OK;
    // a CTA per row is the faster one while its rows leave SMs idle, and where a row is long
    if (rows >= 4 * (int64_t)dev->sm_count && cols <= SM_MAX_COLS) {
        cc_launch_pdl(dev, softmax_rows_kernel, (unsigned)((rows + SM_WARPS - 1) / SM_WARPS), SM_WARPS * 32, 0, x, rows, (int)cols, dev->exp_lut);
        CC_LAUNCH_CHECK(dev);
        return CC_OK;
    }
    cc_launch_pdl(dev, softmax_kernel, (unsigned)rows, CC_RED_THREADS, 0, x, cols, dev->exp_lut);
    CC_LAUNCH_CHECK(dev);
    return CC_OK;
}

// ---- silu / gelu: primitives/silu.rs:6-13, gelu.rs:10-15 -----------------------------------------------------
__global__ void silu_kernel(float* x, int64_t n, const uint16_t* __restrict__ lut) {
    pdl_enter();
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        float v = x[i];
        x[i] = v / (1.0f + exp_cached(-v, lut));
    }
}
__global__ void gelu_kernel(float* x, int64_t n, const uint16_t* __restrict__ lut) {
    pdl_enter();
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) x[i] = h2f_bits(lut[f2h_bits(x[i])]);
}
int cc_launch_silu(cc_device* dev, float* x, int64_t n) {
    if (n == 0) return CC_OK;
    cc_launch_pdl(dev, silu_kernel, (unsigned)((n + 255) / 256), 256, 0, x, n, dev->exp_lut);
    CC_LAUNCH_CHECK(dev);
    return CC_OK;
}
int cc_launch_gelu(cc_device* dev, float* x, int64_t n) {
    if (n == 0) return CC_OK;
    cc_launch_pdl(dev, gelu_kernel, (unsigned)((n + 255) / 256), 256, 0, x, n, dev->gelu_lut);
    CC_LAUNCH_CHECK(dev);
    return CC_OK;
}

// ---- add / mul with rhs cycling: primitives/arithmetic.rs:5-68 ---------------------------------------------------
__global__ void binary_kernel(float* x, int64_t n, const float* __restrict__ y, int64_t ny, int op) {
    pdl_enter();
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float b = y[ny == 1 ? 0 : i % ny];
    x[i] = op == 0 ? x[i] + b : x[i] * b;
}
int cc_launch_binary(cc_device* dev, float* x, int64_t n, const float* y, int64_t ny, int op) {
    if (n == 0) return CC_OK;
    cc_launch_pdl(dev, binary_kernel, (unsigned)((n + 255) / 256), 256, 0, x, n, y, ny, op);
    CC_LAUNCH_CHECK(dev);
    return CC_OK;
}
__global__ void scale_kernel(float* x, int64_t n, float s) {
    pdl_enter();
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) x[i] = x[i] * s;
}
int cc_launch_scale(cc_device* dev, float* x, int64_t n, float s) {     // cpu_tensor.rs:404-410
    if (n == 0) return CC_OK;
    cc_launch_pdl(dev, scale_kernel, (unsigned)((n + 255) / 256), 256, 0, x, n, s);
    CC_LAUNCH_CHECK(dev);
    return CC_OK;
}

// ---- strided copy: contiguous (contiguous.rs:6-66) and concatenate (concatenate.rs:12-77,143-204) ----------------
struct CopyDims { int64_t shape[CC_MAX_DIMS], sstr[CC_MAX_DIMS], dstr[CC_MAX_DIMS]; int ndim; };

__global__ void strided_copy_kernel(const void* src, int src_dtype, void* dst, int dst_dtype, CopyDims d, int64_t dst_offset, int64_t total) {
    pdl_enter();
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    int64_t rem = i, so = 0, dof = dst_offset;
    for (int ax = d.ndim - 1; ax >= 0; ax--) {
        int64_t c = rem % d.shape[ax];
        rem /= d.shape[ax];
        so += c * d.sstr[ax];
        dof += c * d.dstr[ax];
    }
    if (src_dtype == CC_F32 && dst_dtype == CC_F32) ((float*)dst)[dof] = ((const float*)src)[so];
    else if (src_dtype == CC_F16 && dst_dtype == CC_F16) ((__half*)dst)[dof] = ((const __half*)src)[so];
    else if (src_dtype == CC_F32 && dst_dtype == CC_F16) ((__half*)dst)[dof] = __float2half_rn(((const float*)src)[so]);   // f16::from_f32
    else ((float*)dst)[dof] = __half2float(((const __half*)src)[so]);
}
// the case of every cache append and head turn: f32 to f32, rows of unit stride, whose starts are 16-byte aligned on both sides -- a thread moves 16 bytes and
// finds its place with 32-bit divisions.  [512, 32, 128] -> [32, 512, 128] (8 MB): 35 -> 6 us
struct CopyDims32 { unsigned shape[CC_MAX_DIMS], sstr[CC_MAX_DIMS], dstr[CC_MAX_DIMS]; int ndim; };      // last axis and strides in units of 4 elements
__global__ void __launch_bounds__(256) strided_copy16_kernel(const float4* __restrict__ src, float4* __restrict__ dst, CopyDims32 d, unsigned total) {
    pdl_enter();
    const unsigned i = blockIdx.x * 256u + threadIdx.x;
    if (i >= total) return;
    unsigned rem = i, so = 0, dof = 0;
#pragma unroll
    for (int ax = CC_MAX_DIMS - 1; ax >= 0; ax--) {
        if (ax >= d.ndim) continue;
        const unsigned q = rem / d.shape[ax], c = rem - q * d.shape[ax];
        rem = q;
        so += c * d.sstr[ax];
        dof += c * d.dstr[ax];
    }
    dst[dof] = src[so];
}
// whether the copy above may take it; fills d
static bool copy16(const void* src, int src_dtype, const int64_t* sshape, const int64_t* sstrides, const void* dst, int dst_dtype, const int64_t* dstrides, int64_t dst_offset, int ndim,
                   CopyDims32* d) {
    if (src_dtype != CC_F32 || dst_dtype != CC_F32 || ndim < 1 || sstrides[ndim - 1] != 1 || dstrides[ndim - 1] != 1 || sshape[ndim - 1] % 4) return false;
    if ((((uintptr_t)src | (uintptr_t)((const float*)dst + dst_offset)) & 15) != 0) return false;
    int64_t smax = 0, dmax = 0;
    d->ndim = ndim;
    for (int i = 0; i < ndim; i++) {
        if (sstrides[i] < 0 || dstrides[i] < 0) return false;
        if (i + 1 < ndim && sshape[i] > 1 && (sstrides[i] % 4 || dstrides[i] % 4)) return false;
        smax += (sshape[i] - 1) * sstrides[i]; dmax += (sshape[i] - 1) * dstrides[i];
        d->shape[i] = (unsigned)(i + 1 < ndim ? sshape[i] : sshape[i] / 4);
        d->sstr[i] = i + 1 < ndim ? (unsigned)(sstrides[i] / 4) : 1u;
        d->dstr[i] = i + 1 < ndim ? (unsigned)(dstrides[i] / 4) : 1u;
    }
    return smax < ((int64_t)1 << 31) && dmax < ((int64_t)1 << 31);
}
int cc_launch_strided_copy(cc_device* dev, const void* src, int src_dtype, const int64_t* sshape, const int64_t* sstrides,
                           void* dst, int dst_dtype, const int64_t* dstrides, int64_t dst_offset, int ndim) {
    CopyDims d;
    d.ndim = ndim;
    int64_t total = 1;
    for (int i = 0; i < ndim; i++) { d.shape[i] = sshape[i]; d.sstr[i] = sstrides[i]; d.dstr[i] = dstrides[i]; total *= sshape[i]; }
    if (total == 0) return CC_OK;
    CopyDims32 d32;
    if (total < ((int64_t)1 << 31) && copy16(src, src_dtype, sshape, sstrides, dst, dst_dtype, dstrides, dst_offset, ndim, &d32)) {
        const unsigned n = (unsigned)(total / 4);
        cc_launch_pdl(dev, strided_copy16_kernel, (n + 255) / 256, 256, 0, (const float4*)src, (float4*)((float*)dst + dst_offset), d32, n);
        CC_LAUNCH_CHECK(dev);
        return CC_OK;
    }
    cc_launch_pdl(dev, strided_copy_kernel, (unsigned)((total + 255) / 256), 256, 0, src, src_dtype, dst, dst_dtype, d, dst_offset, total);
    CC_LAUNCH_CHECK(dev);
    return CC_OK;
}

// ---- batch_matmul: primitives/batch_matmul.rs:15-131 -----------------------------------------------------------------
// A dense (ab,m,k); B (bb,k,n) strided with stride_k == 1 (K^T view) or stride_n == 1 (V).
// F32 B: kv head = bi % bb (batch_matmul.rs:63);  F16 B: kv head = bi / (ab/bb) (batch_matmul.rs:89-91).
// (a) stride_k == 1: one warp per output, lanes stride over k
template <bool B_F16>
__global__ void bmm_kcontig_kernel(const float* __restrict__ a, const void* __restrict__ b, float* __restrict__ c,
                                   int64_t ab, int64_t bb, int64_t m, int64_t k, int64_t n, int64_t sb0, int64_t sb2) {
    pdl_enter();
    int64_t o = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    int lane = threadIdx.x & 31;
    if (o >= ab * m * n) return;
    int64_t ni = o % n, mi = (o / n) % m, bi = o / (m * n);
    const float* pa = a + bi * (m * k) + mi * k;
    float acc = 0.0f;
    if (B_F16) {
        // A -> f16 (quantize_f32_f16), products and accumulation in f32 (vec_dot_f16_f16_fallback, buf_f16.rs:84-97)
        const __half* pb = (const __half*)b + (bi / (ab / bb)) * sb0 + ni * sb2;
        for (int64_t ki = lane; ki < k; ki += 32) acc += __half2float(__float2half_rn(pa[ki])) * __half2float(pb[ki]);
    } else {
        const float* pb = (const float*)b + (bi % bb) * sb0 + ni * sb2;
        for (int64_t ki = lane; ki < k; ki += 32) acc += pa[ki] * pb[ki];
    }
    acc = warp_sum(acc);
    if (lane == 0) c[o] = acc;
}
// (b) stride_n == 1: one thread per output column, sequential over k (F16: f16 accumulation in the SAME order
//     as vec_fma_f16_f16, buf_f16.rs:152-163, so the result is bit-exact)
template <bool B_F16>
__global__ void bmm_ncontig_kernel(const float* __restrict__ a, const void* __restrict__ b, float* __restrict__ c,
                                   int64_t ab, int64_t bb, int64_t m, int64_t k, int64_t n, int64_t sb0, int64_t sb1) {
    pdl_enter();
    int64_t o = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (o >= ab * m * n) return;
    int64_t ni = o % n, mi = (o / n) % m, bi = o / (m * n);
    const float* pa = a + bi * (m * k) + mi * k;
    if (B_F16) {
        const __half* pb = (const __half*)b + (bi / (ab / bb)) * sb0 + ni;
        __half acc = __float2half_rn(0.0f);
        for (int64_t ki = 0; ki < k; ki++) acc = __hadd(acc, __hmul(pb[ki * sb1], __float2half_rn(pa[ki])));
        c[o] = __half2float(acc);
    } else {
        const float* pb = (const float*)b + (bi % bb) * sb0 + ni;
        float acc = 0.0f;
        for (int64_t ki = 0; ki < k; ki++) acc += pa[ki] * pb[ki * sb1];     // same order as batch_matmul.rs:60-68
        c[o] = acc;
    }
}
// (c) many rows (a prompt): tiles of 128 x 128 on the tensor cores, 32-bit operands and sums (split_gemm.cuh).  F16 B: A is rounded to f16 first, the
//     products are exact and the sums 32-bit, as in (a).  The f16 SUMS of (b) with F16 B have an order of their own and stay there.
// Tiles: columns (fastest), rows, batch.  A warp per output reads 1 KB for 128 products: 32 heads x 512 x 512 x 128 took 1963 us, and 45 us here
template <bool B_F16, bool N_CONTIG>
struct BmmTile {
    static constexpr int HALVES = 2, N = 128;
    static constexpr bool A_TRANSPOSED = false, B_TRANSPOSED = N_CONTIG, SHARED = false, A_TMA = false, B_TMA = false, SKIP_ZERO = false;
    struct Tile { int steps, m0, n0; const float* a; const void* b; float* c; };
    struct Fixed {};
    struct Shared {};
    typedef const float* ARow;
    typedef const void* BCol;
    const float* a;
    const void* b;
    float* c;
    int ab, bb, m, k, n, a_vec, b_vec;
    int64_t sb0, sb1, sb2;
    __device__ bool tile(int i, int, Tile& t) const {
        const int nt = (n + N - 1) / N, mt = (m + 127) >> 7, rest = (unsigned)i / (unsigned)nt, bi = (unsigned)rest / (unsigned)mt;
        t.n0 = (i - rest * nt) * N; t.m0 = (rest - bi * mt) * 128; t.steps = (k + 63) >> 6;
        t.a = a + (int64_t)bi * m * k; t.c = c + (int64_t)bi * m * n;
        if (B_F16) t.b = (const __half*)b + (int64_t)(bi / (ab / bb)) * sb0;
        else t.b = (const float*)b + (int64_t)(bi % bb) * sb0;
        return true;
    }
    __device__ Fixed fixed(int) const { return Fixed{}; }
    __device__ void setup(const Tile&, Shared&) const {}
    __device__ const void* map_a() const { return nullptr; }
    __device__ const void* map_b() const { return nullptr; }
    __device__ void at_a(const Tile&, int, int, int&, int&) const {}
    __device__ void at_b(const Tile&, int, int, int&, int&) const {}
    __device__ ARow a_row(const Tile& t, const Shared&, Fixed, int r) const { return t.m0 + r < m ? t.a + (int64_t)(t.m0 + r) * k : nullptr; }
    __device__ void load_a(const Tile&, ARow p, int s, int ch, float (&v)[8]) const { if (p) sg_load8(p, s * 64 + ch * 8, k, a_vec, v); else sg_zero8(v); }
    __device__ void prep_a(const Tile&, ARow&, float (&v)[8]) const {
        if (!B_F16) return;
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = __half2float(__float2half_rn(v[i]));
    }
    __device__ BCol b_col(const Tile& t, int col) const {
        if (t.n0 + col >= n) return nullptr;
        if (N_CONTIG) return (const float*)t.b + t.n0 + col;
        if (B_F16) return (const __half*)t.b + (int64_t)(t.n0 + col) * sb2;
        return (const float*)t.b + (int64_t)(t.n0 + col) * sb2;
    }
    __device__ void load_b(const Tile&, BCol p, int s, int ch, float (&v)[8]) const {
        const int k0 = s * 64 + ch * 8;
        if (!p) { sg_zero8(v); return; }
        if (N_CONTIG) {
            const float* at = (const float*)p + (int64_t)k0 * sb1;
#pragma unroll
            for (int i = 0; i < 8; i++) { v[i] = k0 + i < k ? *at : 0.0f; at += sb1; }
        } else if (B_F16) {
            const __half* at = (const __half*)p + k0;
            if (b_vec && k0 + 8 <= k) {
                const uint4 h = *(const uint4*)at;
                const unsigned u[4] = {h.x, h.y, h.z, h.w};
#pragma unroll
                for (int i = 0; i < 4; i++) { v[2 * i] = h2f_bits((uint16_t)(u[i] & 0xffffu)); v[2 * i + 1] = h2f_bits((uint16_t)(u[i] >> 16)); }
            } else {
#pragma unroll
                for (int i = 0; i < 8; i++) v[i] = k0 + i < k ? __half2float(at[i]) : 0.0f;
            }
        } else sg_load8((const float*)p, k0, k, b_vec, v);
    }
    __device__ void end_a(const Tile&, Shared&, ARow&, int, int) const {}
    __device__ void give(const Shared&, Shared&, int) const {}
    template <int COUNT>
    __device__ void emit(const Tile& t, const Shared&, Fixed, int r, int col0, float (&v)[COUNT], float* buf) const {
        sg_store_rows<COUNT, false>(buf, t.m0 + r < m ? t.c + (int64_t)(t.m0 + r) * n + t.n0 + col0 : nullptr, n - t.n0 - col0, n % 4 == 0, v);
    }
};
template <bool B_F16, bool N_CONTIG>
static int launch_bmm_tiles(cc_device* dev, const float* a, const void* b, float* c, int64_t ab, int64_t bb, int64_t m, int64_t k, int64_t n, int64_t sb0, int64_t sb1, int64_t sb2) {
    BmmTile<B_F16, N_CONTIG> p{};
    p.a = a; p.b = b; p.c = c; p.ab = (int)ab; p.bb = (int)bb; p.m = (int)m; p.k = (int)k; p.n = (int)n; p.sb0 = sb0; p.sb1 = sb1; p.sb2 = sb2;
    const int per = B_F16 ? 8 : 4;                            // elements of 16 bytes
    p.a_vec = k % 4 == 0 && ((uintptr_t)a & 15) == 0;
    p.b_vec = sb0 % per == 0 && sb2 % per == 0 && ((uintptr_t)b & 15) == 0;
    return sg_launch(dev, p, ((n + 127) / 128) * ((m + 127) / 128) * ab);
}
int cc_launch_batch_matmul(cc_device* dev, const float* a, const void* b, int b_dtype, float* c, int64_t ab, int64_t bb,
                           int64_t m, int64_t k, int64_t n, int64_t sb0, int64_t sb1, int64_t sb2) {
    int64_t outs = ab * m * n;
    if (outs == 0) return CC_OK;
    bool f16 = b_dtype == CC_F16;
    // one row per batch entry (decoding) keeps the order of the fused kernels; the reference's order stays in exact mode.  From 16 rows on a tile that
    // is mostly padding is still faster than reading B once per row
    if (!dev->exact && m >= 16 && k > 0 && ab < 65536 && m < ((int64_t)1 << 24) && n < ((int64_t)1 << 24) && k < ((int64_t)1 << 24) && (sb1 == 1 || !f16)) {
        if (sb1 == 1) return f16 ? launch_bmm_tiles<true, false>(dev, a, b, c, ab, bb, m, k, n, sb0, sb1, sb2) : launch_bmm_tiles<false, false>(dev, a, b, c, ab, bb, m, k, n, sb0, sb1, sb2);
        return launch_bmm_tiles<false, true>(dev, a, b, c, ab, bb, m, k, n, sb0, sb1, sb2);
    }
    if (sb1 == 1) {
        unsigned grid = (unsigned)((outs * 32 + 255) / 256);
        if (f16) cc_launch_pdl(dev, bmm_kcontig_kernel<true>, grid, 256, 0, a, b, c, ab, bb, m, k, n, sb0, sb2);
        else cc_launch_pdl(dev, bmm_kcontig_kernel<false>, grid, 256, 0, a, b, c, ab, bb, m, k, n, sb0, sb2);
    } else {
        unsigned grid = (unsigned)((outs + 127) / 128);
        if (f16) cc_launch_pdl(dev, bmm_ncontig_kernel<true>, grid, 128, 0, a, b, c, ab, bb, m, k, n, sb0, sb1);
        else cc_launch_pdl(dev, bmm_ncontig_kernel<false>, grid, 128, 0, a, b, c, ab, bb, m, k, n, sb0, sb1);
    }
    CC_LAUNCH_CHECK(dev);
    return CC_OK;
}

// ---- greedy sampling on the device: sampler.rs:109-116 (`max_by` keeps the LAST maximum; NaN never wins) -------------------------
// one CTA; thread t scans t, t + 512, ...; ties resolve to the larger index at every level, so the result is the last maximum
__device__ __forceinline__ void argmax_merge(float& bv, long long& bi, float ov, long long oi) {
    if (oi >= 0 && (bi < 0 || ov > bv || (ov == bv && oi > bi))) { bv = ov; bi = oi; }
}
__global__ void __launch_bounds__(CC_RED_THREADS) argmax_kernel(const float* __restrict__ x, long long n, long long* slot, long long* hist,
                                                               const long long* hist_index_dev, long long hist_index) {
    pdl_enter();
    __shared__ float sv[CC_RED_WARPS];
    __shared__ long long si[CC_RED_WARPS];
    float bv = 0.0f; long long bi = -1;
    for (long long i = threadIdx.x; i < n; i += CC_RED_THREADS) { const float v = x[i]; if (bi < 0 || !(v < bv)) { bv = v; bi = i; } }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
        const long long oi = __shfl_xor_sync(0xffffffffu, bi, o);
        argmax_merge(bv, bi, ov, oi);
    }
    if ((threadIdx.x & 31) == 0) { sv[threadIdx.x >> 5] = bv; si[threadIdx.x >> 5] = bi; }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < CC_RED_WARPS; w++) argmax_merge(bv, bi, sv[w], si[w]);
        if (bi < 0) bi = 0;
        *slot = bi;
        const long long h = hist_index_dev ? *hist_index_dev : hist_index;
        if (hist && h >= 0 && h < CC_HISTORY_CAP) hist[h] = bi;
    }
}
int cc_launch_argmax(cc_device* dev, const float* x, int64_t n, int64_t* slot, int64_t* hist, const int64_t* hist_index_dev, int64_t hist_index) {
    cc_launch_pdl(dev, argmax_kernel, 1, CC_RED_THREADS, 0, x, (long long)n, (long long*)slot, (long long*)hist, (const long long*)hist_index_dev, (long long)hist_index);
    CC_LAUNCH_CHECK(dev);
    return CC_OK;
}
