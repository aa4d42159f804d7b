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
    stage_wait();
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
// It takes Q8_0, Q4_0, Q5_K and Q6_K, and of Q4_K up to 4 rows or rows so long that the kernel below has no room for them.  Q4_K, 11008 x 4096, 8 rows: one row at a time
// 58 us, this way 31.  Bound by the integer dot products and the activation reads from shared memory (a 16-byte weight chunk meets 2 x NB 16-byte activation chunks)
template <class T, int NB>
__global__ void __launch_bounds__(MV_THREADS) matvec_few_kernel(WPlanes W, const void* act, int64_t n_total, float* __restrict__ out, int m, int k, int b) {
    pdl_enter();
    extern __shared__ __align__(16) uint8_t smem[];
    const int b0 = blockIdx.y * NB, stride = T::smem_bytes(k);
    for (int n = 0; n < NB; n++) T::stage_act(act, n_total, min(b0 + n, b - 1), k, smem + n * stride);       // activations behind the last repeat it
    stage_wait();
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
// The same for Q4_K on the integer tensor cores.  An mma of 16 x 8 x 16 sums the 16 weights of a chunk's nibbles for 16 weight rows and 8 activations: exactly the
// integers of vecdot.cuh, whose terms follow from them in the same order.  There a lane (super-block mod 4, chunk) adds up its terms and the
// butterfly the lanes; here warp q of four has the super-blocks q, q + 4, .. of the 16 rows and a sum for each of the 8 chunks, and the four warps' sums are
// added up in shared memory in the butterfly's order: identical bits.  A lane holds the weights of two rows at 4 columns of a chunk; activations come by ldmatrix.
// A warp copies its super-blocks (16 rows x 144 B, which lie in memory as in shared memory) four ahead by cp.async (two, where activations of 67 to 73 super-blocks leave no
// more room); rows of 144 B put the words of eight rows in different banks.  One CTA of two groups of four warps an SM.  Half of the
// issue slots are busy (51 %: 707 warp instructions per 16 rows and super-block, the mma among them, two warps a scheduler), the rest are their latencies; more warps only
// stage later (two CTAs an SM 11008 x 4096 x 8 25.1 us, CTAs of 3 / 4 / 5 groups 24.0 / 27.1 / 21.8).
// us with the quantisation of the rows, 11008 x 4096 x 8 / 16 / 31 rows: two weight rows a warp by dp4a 31.4 / 44.1 / 74.2 ; weights by 4-byte loads one super-block ahead and activations
// staged one after another 28.0 / 37.3 / 54.3 ; here 18.8 / 28 / 49.5 ; 32000 x 4096 48 / 72 / 128, now 37 / 67 / 128 ; 4096 x 4096 x 8 17.7, now 10.4.  Q6_K the same
// way: 31.6 by dp4a, 43.4 (its numbers take twice the instructions to put together).
#define MM_THREADS 256
#define MM_GROUPS (MM_THREADS / 128)
#define MM_OUT 128                         // outputs of four warps: 16 rows x 8 activations
#define MM_SB 2304                         // a super-block of 16 rows
__device__ __forceinline__ void mm_mma(int (&c)[4], unsigned a0, unsigned a1, unsigned b) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5}, {%6}, {%0, %1, %2, %3};"
                 : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
                 : "r"(a0), "r"(a1), "r"(b));
}
// one super-block of a lane's two rows (their copies in shared memory) against 8 activations: acc[chunk][output]
struct MmBlock {
    const uint8_t *ra, *rb;                // row lane / 4 and the one 8 behind it
    int c;
    __device__ __forceinline__ void add(float (&acc)[8][4], const unsigned (&b)[16], const uint8_t* const (&act)[2], int k, int sb) const {
        unsigned s[2][2], mn[2][2];
        float d[4], dm[4];
        const int4 h[2] = {*(const int4*)ra, *(const int4*)rb};
        int4 bs[2][2];                                           // block sums of the two activations, two 16-bit numbers a word
#pragma unroll
        for (int n = 0; n < 2; n++) {
            KAct A(act[n], k);
            const int4* at = (const int4*)(A.bs + sb * 16);
            bs[n][0] = at[0]; bs[n][1] = at[1];
            const float da = A.d[sb];
#pragma unroll
            for (int r = 0; r < 2; r++) {
                d[r * 2 + n] = h2f_bits((uint16_t)(h[r].x & 0xFFFF)) * da;
                dm[r * 2 + n] = h2f_bits((uint16_t)((unsigned)h[r].x >> 16)) * da;
            }
        }
#pragma unroll
        for (int r = 0; r < 2; r++) k4_unpack((unsigned)h[r].y, (unsigned)h[r].z, (unsigned)h[r].w, s[r][0], s[r][1], mn[r][0], mn[r][1]);
#pragma unroll
        for (int j = 0; j < 8; j++) {
            int lo[4] = {0, 0, 0, 0}, hi[4] = {0, 0, 0, 0}, sums[2];
            const unsigned w0 = *(const unsigned*)(ra + 16 + 16 * j + 4 * c), w1 = *(const unsigned*)(rb + 16 + 16 * j + 4 * c);
            mm_mma(lo, w0 & 0x0F0F0F0Fu, w1 & 0x0F0F0F0Fu, b[j]);
            mm_mma(hi, (w0 >> 4) & 0x0F0F0F0Fu, (w1 >> 4) & 0x0F0F0F0Fu, b[8 + j]);
            const int g = j >> 1;
#pragma unroll
            for (int n = 0; n < 2; n++) {
                const int4 v = bs[n][j >> 2];
                const int x = (j & 3) == 0 ? v.x : (j & 3) == 1 ? v.y : (j & 3) == 2 ? v.z : v.w;
                sums[n] = (int)(int16_t)(x & 0xFFFF) + (x >> 16);
            }
#pragma unroll
            for (int o = 0; o < 4; o++) {
                const int r = o >> 1, n = o & 1;
                const int isum = byte_of(s[r][0], s[r][1], 2 * g) * lo[o] + byte_of(s[r][0], s[r][1], 2 * g + 1) * hi[o], msum = sums[n] * byte_of(mn[r][0], mn[r][1], j);
                acc[j][o] += d[o] * (float)isum - dm[o] * (float)msum;
            }
        }
    }
};
// distance of two activations in shared memory: an odd number of 16-byte pieces, so that 8 of them lie in different banks
__host__ __device__ __forceinline__ int mm_stride(int bytes) { return (bytes & 16) ? bytes : bytes + 16; }
// shared memory: 8 activations | the warps' super-blocks, S a warp; behind a tile's last one: the warps' sums [groups][4 warps][8 chunks][MM_OUT]
template <int S>
__global__ void __launch_bounds__(MM_THREADS, 1) matvec_mma_kernel(WPlanes W, const void* act, int64_t n_total, float* __restrict__ out, int m, int k, int b) {
    pdl_enter();
    extern __shared__ __align__(16) uint8_t smem[];
    const int b0 = blockIdx.y * 8, there = min(8, b - b0), stride = mm_stride(TQ45_K<false>::smem_bytes(k)), nsb = k >> 8;
    float* part = (float*)(smem + 8 * stride);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, q = warp & 3, group = warp >> 2, c = lane & 3;
    uint8_t* ring = smem + 8 * stride + warp * (S * MM_SB);
    const int nq = (nsb - q + 3) >> 2;                                         // this warp's super-blocks of a tile: q, q + 4, ..
    auto ask = [&](int row0, int i) {                                          // the i-th of them; a group every time, empty behind the last
        if (row0 < m && i < nq) {
            const unsigned to = (unsigned)__cvta_generic_to_shared(ring + (i % S) * MM_SB) + lane * 16;
#pragma unroll
            for (int p = 0; p < 5; p++) {
                const int x = lane + 32 * p, row = x / 9;                      // 9 pieces of 16 B a row
                if (x < 144) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + 512 * p), "l"(W.p[0] + ((int64_t)min(row0 + row, m - 1) * nsb + q + 4 * i) * 144 + (x - 9 * row) * 16) : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int n = 0; n < there; n++) TQ45_K<false>::stage_act(act, n_total, b0 + n, k, smem + n * stride);       // (columns behind the last read it: eight copies of one row made 600 requests a line)
    asm volatile("cp.async.commit_group;" ::: "memory");
    for (int i = 0; i < S; i++) ask((int)(blockIdx.x * MM_GROUPS + group) * 16, i);
    asm volatile("cp.async.wait_group %0;" ::"n"(S) : "memory");              // the activations
    __syncthreads();
    const uint8_t* const mine[2] = {smem + min(2 * c, there - 1) * stride, smem + min(2 * c + 1, there - 1) * stride};      // the activations of this lane's outputs
    const unsigned rows = (unsigned)__cvta_generic_to_shared(smem + min(lane & 7, there - 1) * stride) + ((lane & 8) ? 128 : 0) + ((lane & 16) ? 16 : 0);      // ldmatrix: chunks j, j + 8, j + 1, j + 9
    for (int t = blockIdx.x; t * (16 * MM_GROUPS) < m; t += gridDim.x) {
        const int row0 = (t * MM_GROUPS + group) * 16;
        float acc[8][4];
#pragma unroll
        for (int j = 0; j < 8; j++) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.0f;
        if (row0 < m) {
#pragma unroll 1
            for (int i = 0; i < nq; i++) {
                const int sb = q + 4 * i;
                unsigned bx[16];
#pragma unroll
                for (int j = 0; j < 8; j += 2)
                    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(bx[j]), "=r"(bx[8 + j]), "=r"(bx[j + 1]), "=r"(bx[9 + j]) : "r"(rows + sb * 256 + j * 16));
                asm volatile("cp.async.wait_group %0;" ::"n"(S - 1) : "memory");
                __syncwarp();
                MmBlock blk;
                blk.ra = ring + (i % S) * MM_SB + (lane >> 2) * 144; blk.rb = blk.ra + 8 * 144; blk.c = c;
                blk.add(acc, bx, mine, k, sb);
                __syncwarp();
                ask(row0, i + S);
            }
        }
        __syncthreads();                                                       // the sums go where the super-blocks were
        float* to = part + ((group * 4 + q) * 8) * MM_OUT + lane * 4;
#pragma unroll
        for (int j = 0; j < 8; j++) *(float4*)(to + j * MM_OUT) = make_float4(acc[j][0], acc[j][1], acc[j][2], acc[j][3]);
        __syncthreads();
        const int o = threadIdx.x & (MM_OUT - 1);                              // output o of this thread's group: lane o / 4, number o % 4 of it
        const float* from = part + (threadIdx.x / MM_OUT) * (32 * MM_OUT) + o;
        float v[8];
#pragma unroll
        for (int j = 0; j < 8; j++) v[j] = (from[j * MM_OUT] + from[(16 + j) * MM_OUT]) + (from[(8 + j) * MM_OUT] + from[(24 + j) * MM_OUT]);
        const float sum = ((v[0] + v[4]) + (v[2] + v[6])) + ((v[1] + v[5]) + (v[3] + v[7]));
        const int row = (t * MM_GROUPS + (int)threadIdx.x / MM_OUT) * 16 + (o >> 4) + ((o & 2) ? 8 : 0), n = b0 + ((o >> 2) & 3) * 2 + (o & 1);
        if (row < m && n < b) out[(int64_t)n * m + row] = sum;
        if ((t + (int)gridDim.x) * (16 * MM_GROUPS) < m) {
            __syncthreads();
            for (int i = 0; i < S; i++) ask(row0 + (int)gridDim.x * (16 * MM_GROUPS), i);
        }
    }
}
static int mm_act_bytes(int64_t k) { return 8 * mm_stride(TQ45_K<false>::smem_bytes((int)k)); }
static int mm_smem(int64_t k, int stages) { const int part = MM_GROUPS * 32 * MM_OUT * 4, ring = MM_GROUPS * 4 * stages * MM_SB; return mm_act_bytes(k) + (part > ring ? part : ring); }
#define MM_MOST (224 * 1024)
static bool mm_fits(int64_t k) { return mm_act_bytes(k) <= 168 * 1024; }
template <int S>
static int launch_mma_as(cc_device* dev, const WPlanes& W, const void* act, int64_t n_total, float* out, int64_t m, int64_t k, int64_t b, int64_t ctas) {
    int smem = mm_smem(k, S);
    // an SM for each CTA: more than half of its shared memory.  Started while the kernel before is still there, some SMs took two and others none
    if (smem < 116 * 1024) smem = 116 * 1024;
    CC_CUDA(dev, cudaFuncSetAttribute(matvec_mma_kernel<S>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    cc_launch_pdl(dev, matvec_mma_kernel<S>, dim3((unsigned)ctas, (unsigned)((b + 7) / 8)), MM_THREADS, smem, W, act, n_total, out, (int)m, (int)k, (int)b);
    CC_LAUNCH_CHECK(dev);
    return CC_OK;
}
static int launch_mma(cc_device* dev, const cc_buf* w, const void* act, int64_t n_total, float* out, int64_t m, int64_t k, int64_t b) {
    WPlanes W;
    for (int i = 0; i < CC_MAX_PLANES; i++) W.p[i] = w->plane[i];
    const int64_t groups = (b + 7) / 8, most = dev->sm_count / groups > 0 ? dev->sm_count / groups : 1, tiles = (m + 16 * MM_GROUPS - 1) / (16 * MM_GROUPS), ctas = tiles < most ? tiles : most;
    return mm_smem(k, 4) <= MM_MOST ? launch_mma_as<4>(dev, W, act, n_total, out, m, k, b, ctas) : launch_mma_as<2>(dev, W, act, n_total, out, m, k, b, ctas);
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
    case CC_Q4_K:
        // (up to 4 rows the dp4a kernel: 11008 x 4096, 4 rows 20.1 us by it, 25.5 here ; from 5 on it takes 8 rows' time for each 8: 31.4 and 27.3)
        if (b > 4 && mm_fits(k)) return launch_mma(dev, w, act, n_total, out, m, k, b);
        return launch_rows<TQ45_K<false>>(dev, w, act, n_total, out, m, k, b);
    case CC_Q5_K: return launch_rows<TQ45_K<true>>(dev, w, act, n_total, out, m, k, b);
    case CC_Q6_K: return launch_rows<TQ6_K>(dev, w, act, n_total, out, m, k, b);
    case CC_Q8_K: return launch<TQ8_K>(dev, w, act, n_total, out, m, k, b);
    }
    return cc_fail(dev, CC_ERR_UNSUPPORTED, "matmul_vec: weight type %d is not supported", w->dtype);
}
