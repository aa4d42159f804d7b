// matvec.cu -- THE hot path: C[b,m] = sum_k W[m,k] * x[b,k] with W in GGUF quant blocks
// (reference: primitives/matmul_vec.rs:26-78 -> buf/buf_q*.rs vec_dot_*).
//
// Design (HBM-bound integer/byte work -- no tensor cores on purpose):
//   * one warp per output row; weight bytes are streamed exactly once with 16-byte LDG.128
//     (L1::no_allocate), consecutive lanes read consecutive 16-byte chunks -> 512 B per warp request;
//   * the quantised activation (Q8_0 / Q8_1 / Q8_K, a few KB) is staged once per CTA in shared memory;
//   * in-register unpack (nibble / high-bit / 2-bit fields), dp4a integer dots, one f32 scale
//     multiply per block, warp-shuffle reduction;
//   * integer sub-block sums are exact; only the order of the final f32 accumulation differs
//     from the reference's scalar loops (tolerance 1e-5 rel in tests/test_gpu_matvec.py).
#include "common.cuh"
#include "vecdot.cuh"

#define MV_THREADS 256
#define MV_WARPS (MV_THREADS / 32)

template <class T>
__global__ void __launch_bounds__(MV_THREADS) matvec_kernel(WPlanes W, const void* act, int64_t n_total,
                                                            float* __restrict__ out, int m, int k) {
    pdl_enter();
    extern __shared__ __align__(16) uint8_t smem[];
    const int bi = blockIdx.y;
    T::stage_act(act, n_total, bi, k, smem);
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int row = blockIdx.x * MV_WARPS + warp; row < m; row += gridDim.x * MV_WARPS) {
        float acc = T::row_dot(W, row, k, smem, lane);
        acc = warp_sum(acc);
        if (lane == 0) out[(int64_t)bi * m + row] = acc;
    }
}

// a few activation rows (2 .. 31: several sequences' next tokens): the grid above fetches and unpacks the weights once per row.  Here a warp takes two weight
// rows and NB activations at a time (vecdot.cuh rows_dot); a CTA stages its NB activations once and walks over the weight rows.
// Q4_K, 11008 x 4096, 8 rows: 58 -> 37 us (whole call 77 -> 48) for 25 MB of weights (3.9 us at the copy rate); bound by the integer dot products and the
// activation reads from shared memory (a 16-byte weight chunk meets 2 x NB 16-byte activation chunks)
template <class T, int NB>
__global__ void __launch_bounds__(MV_THREADS) matvec_few_kernel(WPlanes W, const void* act, int64_t n_total, float* __restrict__ out, int m, int k, int b) {
    pdl_enter();
    extern __shared__ __align__(16) uint8_t smem[];
    const int b0 = blockIdx.y * NB, stride = T::smem_bytes(k);
    for (int n = 0; n < NB; n++) T::stage_act(act, n_total, min(b0 + n, b - 1), k, smem + n * stride);       // activations behind the last repeat it
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int row = (blockIdx.x * MV_WARPS + warp) * 2; row < m; row += gridDim.x * MV_WARPS * 2) {
        float acc[2][NB];
#pragma unroll
        for (int n = 0; n < NB; n++) acc[0][n] = acc[1][n] = 0.0f;
        T::template rows_dot<2, NB>(W, row, m, k, smem, stride, lane, acc);
#pragma unroll
        for (int n = 0; n < NB; n++) {
            const float x = warp_sum(acc[0][n]), y = warp_sum(acc[1][n]);
            if (lane < 2 && row + lane < m && b0 + n < b) out[(int64_t)(b0 + n) * m + row + lane] = lane ? y : x;
        }
    }
}
template <class T, int NB>
static int launch_few(cc_device* dev, const WPlanes& W, const void* act, int64_t n_total, float* out, int64_t m, int64_t k, int64_t b) {
    const int smem = NB * T::smem_bytes((int)k);
    if (smem > 48 * 1024) CC_CUDA(dev, cudaFuncSetAttribute(matvec_few_kernel<T, NB>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    const int64_t groups = (b + NB - 1) / NB, need = (m + 2 * MV_WARPS - 1) / (2 * MV_WARPS), most = smem > 100 * 1024 ? dev->sm_count : 2 * (int64_t)dev->sm_count;
    int64_t ctas = most / groups > 0 ? most / groups : 1;
    if (ctas > need) ctas = need;
    cc_launch_pdl(dev, matvec_few_kernel<T, NB>, dim3((unsigned)ctas, (unsigned)groups), MV_THREADS, smem, W, act, n_total, out, (int)m, (int)k, (int)b);
    CC_LAUNCH_CHECK(dev);
    return CC_OK;
}
template <class T>
static int launch(cc_device* dev, const cc_buf* w, const void* act, int64_t n_total, float* out, int64_t m, int64_t k, int64_t b) {
    WPlanes W;
    for (int i = 0; i < CC_MAX_PLANES; i++) W.p[i] = w->plane[i];
    int smem = T::smem_bytes((int)k);
    if (smem > 48 * 1024) {
        CC_REQUIRE(dev, smem <= 200 * 1024, "matmul_vec: k=%lld needs %d bytes of shared memory", (long long)k, smem);
        CC_CUDA(dev, cudaFuncSetAttribute(matvec_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    }
    int64_t ctas = (m + MV_WARPS - 1) / MV_WARPS;
    int64_t cap = (int64_t)dev->sm_count * 8;
    if (ctas > cap) ctas = cap;
    dim3 grid((unsigned)ctas, (unsigned)b);
    cc_launch_pdl(dev, matvec_kernel<T>, grid, MV_THREADS, smem, W, act, n_total, out, (int)m, (int)k);
    CC_LAUNCH_CHECK(dev);
    return CC_OK;
}

// as many activations at a time as there are and as fit; rows too long for two of them stay with a row at a time
template <class T>
static int launch_rows(cc_device* dev, const cc_buf* w, const void* act, int64_t n_total, float* out, int64_t m, int64_t k, int64_t b) {
    const int64_t one = T::smem_bytes((int)k), most = 200 * 1024;
    WPlanes W;
    for (int i = 0; i < CC_MAX_PLANES; i++) W.p[i] = w->plane[i];
    if (b > 4 && 8 * one <= most) return launch_few<T, 8>(dev, W, act, n_total, out, m, k, b);
    if (b > 2 && 4 * one <= most) return launch_few<T, 4>(dev, W, act, n_total, out, m, k, b);
    if (b > 1 && 2 * one <= most) return launch_few<T, 2>(dev, W, act, n_total, out, m, k, b);
    return launch<T>(dev, w, act, n_total, out, m, k, b);
}

int cc_launch_matvec(cc_device* dev, const cc_buf* w, const void* act, const float* x_f32, float* out,
                     int64_t m, int64_t k, int64_t b) {
    if (m == 0 || b == 0) return CC_OK;
    const int64_t n_total = b * k;
    switch (w->dtype) {
    case CC_F32: return launch<TF32>(dev, w, x_f32, n_total, out, m, k, b);
    case CC_F16: return launch<TF16>(dev, w, act, n_total, out, m, k, b);
    case CC_BF16: return launch<TBF16>(dev, w, x_f32, n_total, out, m, k, b);
    case CC_Q8_0: return launch_rows<TQ8_0>(dev, w, act, n_total, out, m, k, b);
    case CC_Q4_0: return launch_rows<TQ4_0>(dev, w, act, n_total, out, m, k, b);
    case CC_Q5_0: return launch<TQ5_0>(dev, w, act, n_total, out, m, k, b);
    case CC_Q4_1: return launch<TQx_1<false>>(dev, w, act, n_total, out, m, k, b);
    case CC_Q5_1: return launch<TQx_1<true>>(dev, w, act, n_total, out, m, k, b);
    case CC_Q2_K: return launch<TQ2_K>(dev, w, act, n_total, out, m, k, b);
    case CC_Q3_K: return launch<TQ3_K>(dev, w, act, n_total, out, m, k, b);
    case CC_Q4_K: return launch_rows<TQ45_K<false>>(dev, w, act, n_total, out, m, k, b);
    case CC_Q5_K: return launch_rows<TQ45_K<true>>(dev, w, act, n_total, out, m, k, b);
    case CC_Q6_K: return launch_rows<TQ6_K>(dev, w, act, n_total, out, m, k, b);
    case CC_Q8_K: return launch<TQ8_K>(dev, w, act, n_total, out, m, k, b);
    }
    return cc_fail(dev, CC_ERR_UNSUPPORTED, "matmul_vec: weight type %d is not supported", w->dtype);
}
