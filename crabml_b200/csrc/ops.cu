// ops.cu -- the small ops around the matvec, one launch per trait call.
// Compiled with -fmad=false / IEEE div+sqrt so that every op reproduces the reference's f32
// arithmetic; only reduction ORDER differs (the canonical 512-thread tree of common.cuh instead of sequential).
#include "common.cuh"

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
// 16 bytes a thread: [32, 512, 128] 10.6 us by single numbers, 5.1.  Call after call it takes 1.05 million numbers 4.6 and 3.9 us; below that a call waits for the
// host, whose launch of this kernel takes 0.4 us longer (512 numbers 3.8 and 4.3 us), so a decoded token's few thousand go by single numbers
#define SCALE4_FROM ((int64_t)1 << 19)
__global__ void __launch_bounds__(256) scale4_kernel(float4* x, unsigned n4, float s) {
    pdl_enter();
    const unsigned i = blockIdx.x * 256u + threadIdx.x;
    if (i >= n4) return;
    const float4 v = x[i];
    x[i] = make_float4(v.x * s, v.y * s, v.z * s, v.w * s);
}
int cc_launch_scale(cc_device* dev, float* x, int64_t n, float s) {     // cpu_tensor.rs:404-410
    if (n == 0) return CC_OK;
    if (n >= SCALE4_FROM && n % 4 == 0 && n < ((int64_t)1 << 32) && ((uintptr_t)x & 15) == 0) {
        cc_launch_pdl(dev, scale4_kernel, (unsigned)((n / 4 + 255) / 256), 256, 0, (float4*)x, (unsigned)(n / 4), s);
        CC_LAUNCH_CHECK(dev);
        return CC_OK;
    }
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
// two 32-bit numbers an instruction, each rounded as by itself.  nz: two times -0, which changes no product, as a value that the assembler does not know: it makes one
// instruction with one rounding of a mul.rn.f32x2 (or an fma with a constant) and the addition behind it
__device__ __forceinline__ uint64_t two(float a, float b) { uint64_t v; asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b)); return v; }
__device__ __forceinline__ float2 apart(uint64_t v) { float2 x; asm("mov.b64 {%0, %1}, %2;" : "=f"(x.x), "=f"(x.y) : "l"(v)); return x; }
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b, uint64_t nz) { uint64_t v; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(v) : "l"(a), "l"(b), "l"(nz)); return v; }
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) { uint64_t v; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b)); return v; }
// (c) many rows: the sums of (a), bit for bit.  A thread makes 4 x 4 outputs of a 64 x 64 tile whose operands lie in shared memory for the whole depth (up to
//     BK_DEPTH), so that it can take the 32 lanes' partial sums in the order in which the butterfly adds them -- lanes 0, 16, 8, 24, 4, .. -- and keep one
//     unfinished sum per level of its tree.  Column k of 64 rows lies in 16 groups of 4, group g at place g ^ (k / 4): rows arrive along k and are read across.
//     32 heads x 512 x 512 x 128, 1.1 G terms of two roundings (60 us at one a lane and cycle): 108 us ; a warp per output reads 1 KB for 128 terms: 1945 us
#define BK_TILE 64
#define BK_DEPTH 384
__device__ __forceinline__ int bk_at(int k, int group) { return k * BK_TILE + ((group ^ ((k >> 2) & 15)) << 2); }
template <bool B_F16>
__global__ void __launch_bounds__(256, 2) bmm_kcontig_tile_kernel(const float* __restrict__ a, const void* __restrict__ b, float* __restrict__ c, int ab, int bb, int m, int k, int n,
                                                                  int64_t sb0, int64_t sb2, int n_tiles, int m_tiles, int a_vec, int b_vec, uint64_t nz) {
    pdl_enter();
    extern __shared__ __align__(16) float bk_sm[];           // [depth][64] of A, [depth][64] of B
    float *sa = bk_sm, *sb = bk_sm + ((k + 3) & ~3) * BK_TILE;
    const int rest = blockIdx.x / (unsigned)n_tiles, bi = rest / m_tiles, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int m0 = (rest - bi * m_tiles) * BK_TILE, n0 = ((int)blockIdx.x - rest * n_tiles) * BK_TILE;
    const float* pa = a + ((int64_t)bi * m + m0) * k;
    const float* pf = (const float*)b + (int64_t)(bi % bb) * sb0 + n0 * sb2;
    const __half* ph = (const __half*)b + (int64_t)(bi / (ab / bb)) * sb0 + n0 * sb2;
    // a warp moves 4 rows x 32 of the depth at a time, rows outside as zeros ; the four runs of rows it has go together
    for (int k0 = (lane >> 2) * 4; k0 < k; k0 += 32) {
        float v[4][4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int r = (warp + (u & 1) * 8) * 4 + (lane & 3);
            const bool left = u < 2, on = left ? m0 + r < m : n0 + r < n;
            if (on && (left || !B_F16)) {
                const float* p = left ? pa + (int64_t)r * k + k0 : pf + r * sb2 + k0;
                if (left ? a_vec : b_vec) { const float4 x = *(const float4*)p; v[u][0] = x.x; v[u][1] = x.y; v[u][2] = x.z; v[u][3] = x.w; }
                else {
#pragma unroll
                    for (int i = 0; i < 4; i++) v[u][i] = k0 + i < k ? p[i] : 0.0f;
                }
            } else {
#pragma unroll
                for (int i = 0; i < 4; i++) v[u][i] = on && k0 + i < k ? __half2float(ph[r * sb2 + k0 + i]) : 0.0f;
            }
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
            float* to = (u < 2 ? sa : sb) + bk_at(k0, warp + (u & 1) * 8) + (lane & 3);
#pragma unroll
            for (int i = 0; i < 4; i++) to[i * BK_TILE] = B_F16 && u < 2 ? __half2float(__float2half_rn(v[u][i])) : v[u][i];
        }
    }
    __syncthreads();
    const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15, row0 = m0 + ty * 4, col0 = n0 + tx * 4;
    if (m0 + (warp * 2) * 4 >= m) return;                    // none of the warp's rows
    uint64_t tree[5][8], sum[8];                             // [2 j + i]: rows 2 i and 2 i + 1 of column j
#pragma unroll
    for (int t = 0; t < 32; t++) {
        const int l = (t & 1) << 4 | (t & 2) << 2 | (t & 4) | (t & 8) >> 2 | (t & 16) >> 4;
#pragma unroll
        for (int i = 0; i < 8; i++) sum[i] = 0;
        // places of two steps of 32 differ in one bit of the group
        const float *a0 = sa + bk_at(l, ty), *a1 = sa + bk_at(l + 32, ty), *b0 = sb + bk_at(l, tx), *b1 = sb + bk_at(l + 32, tx);
        for (int ki = l; ki < k; ki += 64) {
            const ulonglong2 x = *(const ulonglong2*)a0;
            const float4 y = *(const float4*)b0;
            const uint64_t xr[2] = {x.x, x.y}, yr[4] = {two(y.x, y.x), two(y.y, y.y), two(y.z, y.z), two(y.w, y.w)};
#pragma unroll
            for (int i = 0; i < 8; i++) sum[i] = add2(sum[i], mul2(xr[i & 1], yr[i >> 1], nz));
            if (ki + 32 < k) {
                const ulonglong2 x1 = *(const ulonglong2*)a1;
                const float4 y1 = *(const float4*)b1;
                const uint64_t xs[2] = {x1.x, x1.y}, ys[4] = {two(y1.x, y1.x), two(y1.y, y1.y), two(y1.z, y1.z), two(y1.w, y1.w)};
#pragma unroll
                for (int i = 0; i < 8; i++) sum[i] = add2(sum[i], mul2(xs[i & 1], ys[i >> 1], nz));
            }
            a0 += 64 * BK_TILE; a1 += 64 * BK_TILE; b0 += 64 * BK_TILE; b1 += 64 * BK_TILE;
        }
        int level = 0;
#pragma unroll
        for (; level < 5 && ((t >> level) & 1); level++)
#pragma unroll
            for (int i = 0; i < 8; i++) sum[i] = add2(tree[level][i], sum[i]);
        if (level < 5) {
#pragma unroll
            for (int i = 0; i < 8; i++) tree[level][i] = sum[i];
        }
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        if (row0 + i >= m) break;
        float* o = c + ((int64_t)bi * m + row0 + i) * n + col0;
        float v[4];
#pragma unroll
        for (int j = 0; j < 4; j++) { const float2 x = apart(sum[2 * j + (i >> 1)]); v[j] = i & 1 ? x.y : x.x; }
        if (n % 4 == 0 && col0 < n) *(float4*)o = make_float4(v[0], v[1], v[2], v[3]);
        else {
#pragma unroll
            for (int j = 0; j < 4; j++) if (col0 + j < n) o[j] = v[j];
        }
    }
}
// (d) many rows of (b), F32 B: the same sum per output in one thread, ascending k; 32 x 64 tiles staged 16 deep in two buffers of shared memory, 4 x 4 outputs a
//     thread.  The f16 SUMS of (b) with F16 B stay there.  32 heads x 512 x 128 over 512: 300 -> 79 us
#define BN_ROWS 32
#define BN_TILE 64
#define BN_K 16
__global__ void __launch_bounds__(128) bmm_ncontig_tile_kernel(const float* __restrict__ a, const float* __restrict__ b, float* __restrict__ c, int bb, int m, int k, int n,
                                                               int64_t sb0, int64_t sb1, int n_tiles, int m_tiles, int a_vec, int b_vec, uint64_t nz) {
    pdl_enter();
    __shared__ __align__(16) float sa[2][BN_K][BN_ROWS + 4], sb[2][BN_K][BN_TILE];
    const int rest = blockIdx.x / (unsigned)n_tiles, bi = rest / m_tiles;
    const int m0 = (rest - bi * m_tiles) * BN_ROWS, n0 = ((int)blockIdx.x - rest * n_tiles) * BN_TILE;
    const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
    const int ar = threadIdx.x >> 2, ak = (threadIdx.x & 3) * 4, bk = threadIdx.x >> 3, bn = (threadIdx.x & 7) * 8;      // what a thread stages: 4 of a row of A, 8 of B's
    const float* pa = m0 + ar < m ? a + ((int64_t)bi * m + m0 + ar) * k : nullptr;
    const float* pb = b + (int64_t)(bi % bb) * sb0 + n0;
    float va[4], vb[8];
    uint64_t acc[2][4];                                      // [i][j]: rows 2 i and 2 i + 1 of column j
    auto four = [](const float* p, int at, int end, bool vec, float* v) {      // p[at ..], zeros from `end` on: they add exact zeros
        if (p && vec && at + 4 <= end) {
            const float4 x = *(const float4*)(p + at);
            v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
        } else {
#pragma unroll
            for (int i = 0; i < 4; i++) v[i] = p && at + i < end ? p[at + i] : 0.0f;
        }
    };
    auto fetch = [&](int k0) {
        const float* row = k0 + bk < k ? pb + (int64_t)(k0 + bk) * sb1 : nullptr;
        four(pa, k0 + ak, k, a_vec, va);
        four(row, bn, n - n0, b_vec, vb);
        four(row, bn + 4, n - n0, b_vec, vb + 4);
    };
    auto put = [&](int s) {
#pragma unroll
        for (int i = 0; i < 4; i++) sa[s][ak + i][ar] = va[i];
        *(float4*)&sb[s][bk][bn] = make_float4(vb[0], vb[1], vb[2], vb[3]);
        *(float4*)&sb[s][bk][bn + 4] = make_float4(vb[4], vb[5], vb[6], vb[7]);
    };
#pragma unroll
    for (int i = 0; i < 8; i++) acc[i >> 2][i & 3] = 0;
    fetch(0);
    put(0);
    for (int k0 = 0, s = 0; k0 < k; k0 += BN_K, s ^= 1) {
        __syncthreads();                                                 // this step's operands are there, the last one's have been read
        if (k0 + BN_K < k) fetch(k0 + BN_K);                             // the next step's travel while this one is multiplied
        if (m0 + (int)(threadIdx.x >> 5) * 8 < m) {                      // (a warp has rows 8 w ..)
#pragma unroll
            for (int kk = 0; kk < BN_K; kk++) {
                const ulonglong2 x = *(const ulonglong2*)&sa[s][kk][ty * 4];
                const float4 y = *(const float4*)&sb[s][kk][tx * 4];
                const uint64_t xr[2] = {x.x, x.y}, yr[4] = {two(y.x, y.x), two(y.y, y.y), two(y.z, y.z), two(y.w, y.w)};
#pragma unroll
                for (int i = 0; i < 8; i++) acc[i >> 2][i & 3] = add2(acc[i >> 2][i & 3], mul2(xr[i >> 2], yr[i & 3], nz));
            }
        }
        if (k0 + BN_K < k) put(s ^ 1);
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int row = m0 + ty * 4 + i;
        if (row >= m) break;
        float* o = c + ((int64_t)bi * m + row) * n + n0 + tx * 4;
        float v[4];
#pragma unroll
        for (int j = 0; j < 4; j++) { const float2 x = apart(acc[i >> 1][j]); v[j] = i & 1 ? x.y : x.x; }
        if (n % 4 == 0 && n0 + tx * 4 < n) *(float4*)o = make_float4(v[0], v[1], v[2], v[3]);
        else {
#pragma unroll
            for (int j = 0; j < 4; j++) if (n0 + tx * 4 + j < n) o[j] = v[j];
        }
    }
}
int cc_launch_batch_matmul(cc_device* dev, const float* a, const void* b, int b_dtype, float* c, int64_t ab, int64_t bb,
                           int64_t m, int64_t k, int64_t n, int64_t sb0, int64_t sb1, int64_t sb2) {
    int64_t outs = ab * m * n;
    if (outs == 0) return CC_OK;
    bool f16 = b_dtype == CC_F16;
    // a tile's time does not depend on how many of its rows there are, (a) and (b) go row by row.  us for 1 / 2 / 4 / 8 rows of 32 heads, K = 128, 512 columns: (a) 11, 11,
    // 19, 34 beside 11 in tiles, 2048 columns: 19, 34, 64, 125 beside 38 ; 512 terms, 128 columns: (b) 35 beside 24
    const int64_t m_tiles = sb1 == 1 ? (m + BK_TILE - 1) / BK_TILE : (m + BN_ROWS - 1) / BN_ROWS, n_tiles = (n + 63) / 64;
    if (m >= 4 && (sb1 == 1 ? k <= BK_DEPTH : !f16) && ab < (1 << 24) && m < (1 << 24) && n < (1 << 24) && k < (1 << 24) && m_tiles * n_tiles * ab < ((int64_t)1 << 31)) {
        static_assert(BK_TILE == 64 && BN_TILE == 64, "one count of column tiles");
        const unsigned tiles = (unsigned)(m_tiles * n_tiles * ab);
        const int a_vec = k % 4 == 0 && ((uintptr_t)a & 15) == 0, b_vec = !f16 && ((uintptr_t)b & 15) == 0 && sb0 % 4 == 0 && (sb1 == 1 ? sb2 % 4 == 0 && k % 4 == 0 : sb1 % 4 == 0);
        if (sb1 != 1) cc_launch_pdl(dev, bmm_ncontig_tile_kernel, tiles, 128, 0, a, (const float*)b, c, (int)bb, (int)m, (int)k, (int)n, sb0, sb1, (int)n_tiles, (int)m_tiles, a_vec, b_vec, (uint64_t)0x8000000080000000ull);
        else {
            const int smem = 2 * (int)((k + 3) & ~3) * BK_TILE * 4;
            auto kernel = f16 ? bmm_kcontig_tile_kernel<true> : bmm_kcontig_tile_kernel<false>;
            if (smem > 48 * 1024) CC_CUDA(dev, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
            cc_launch_pdl(dev, kernel, tiles, 256, smem, a, b, c, (int)ab, (int)bb, (int)m, (int)k, (int)n, sb0, sb2, (int)n_tiles, (int)m_tiles, a_vec, b_vec, (uint64_t)0x8000000080000000ull);
        }
        CC_LAUNCH_CHECK(dev);
        return CC_OK;
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
