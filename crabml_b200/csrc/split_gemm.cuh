// split_gemm.cuh -- products of 32-bit operands on the tensor cores without giving up 32 bits.
//
// An operand x is cut into three bfloat16 numbers h + m + l (8 mantissa bits each, each the nearest to what is left, so that all 24 bits are kept), and a
// product is the sum of six of the nine partial products: hh + (hm + mh) + (hl + mm + lh).  With x in [1, 2), |m| <= 2^-8 and |l| <= 2^-17, so that what is
// left out, ml + lm + ll, stays below 2^-24 of the product, of either sign (cut off instead of rounded it reached 2^-21, always of the product's own sign).  tcgen05.mma adds a group of 16
// products to its accumulator and cuts the sum off at 24 bits (measured: 1 + 0.75 ulp stays 1), so a long chain of additions would drift towards
// zero.  Therefore hh has an accumulator of its own that is read out after 128 terms (a run of two steps) and added to a 32-bit register sum with
// ordinary rounding; the other five, 2^-8 and less of it, are read out once.  Where the runs begin is the user's to say (Tile::half): a sum whose first
// terms are zeros in one tile and absent in another keeps its bits when both tiles pair the same steps.  Measured error and speed: at the users of this header.
//
// Why not CUDA cores: 148 SMs x 128 fused multiply-adds at 1.9 GHz are 72 TFLOP/s at the very best; the six bfloat16 products of a 128 x 128 x 64
// step take the tensor core 1536 cycles, which is 380 TFLOP/s of 32-bit product.  The three planes of N columns of B lie one behind the other, so
// four instructions make the six products: A_h x B_h, A_h x [B_m B_l], A_m x [B_h B_m], A_l x B_h.  One instruction per product reads the planes of A
// from shared memory more often; at N = 64 it took 85 cycles for 32 cycles of arithmetic.
//
// B, and A where A_TMA says so, arrive by TMA: a kernel before this one has cut them into planes in global memory (what many tiles read), three boxes of
// 64 columns per step.  Otherwise warps 0-15 load A as 32-bit numbers, cut and store them (128-byte swizzle, K-major) while they are staged.  Cutting costs
// about six instructions per element and a trip through registers: with both operands cut in the kernel, a step of 128 x 128 x 64 took 5400 cycles.
//
// One CTA per SM: warps 0-15 stage and collect, warp 16 issues the products (issuing blocks while the tensor core is busy), warp 17 the TMA loads.  Step
// s: cut this warp's share of 64 columns into one of two stages, issuing the loads of step s + 1 as registers become free; then collect
// the accumulators if step s - 1 closed a run of two.  A CTA walks over the tiles blockIdx.x, blockIdx.x + gridDim.x, ... (SPLIT: the two CTAs of
// a cluster share a tile's steps, and each finishes half of its columns with the sums of both).
// Every wait is bounded: on expiry the CTA raises `fail`, every warp leaves its loop, TMEM is freed and the host reports it.
//
// An infinity cannot be cut (its rest is NaN), nor what rounds to one: sums that come out as NaN are computed again in plain 32-bit arithmetic from the same operands, so
// that infinities spread exactly as far as they would in a sum of products.
//
// The user is a struct P (a kernel argument) with
//   static constexpr int HALVES    a tile has 64 * HALVES columns (1 or 2)
//   struct Tile { int steps, half; ... } bool tile(i, rank, Tile&): the i-th tile, false = nothing to do; steps = ceil(K / 64); SPLIT: those of CTA `rank`;
//                                  half: 1 = the first step is the second of its run
//   Fixed, fixed(r)                what does not change from tile to tile about row r
//   SHARED, Shared                 void setup(Tile, Shared&) is called by all threads before a tile, which then waits for the one before
//   ARow, BCol                     what a thread keeps of a row / a column
//   map_b, at_b (A_TMA: map_a ..)  the tensor map and the coordinates of a step's box of a plane
//   a_row, load_a, prep_a          where A is cut here, and for sums that are computed again: a row of A; 8 consecutive elements of it as they lie in memory;
//   b_col, load_b                  the operand they stand for; a column of B and 8 consecutive elements of it
//   SKIP_ZERO                      in sums that are computed again, a zero of A leaves its term out (weights of masked keys)
//   end_a                          SHARED: after the last step, with the thread's row state
//   emit                           the epilogue: 16 * HALVES consecutive sums of a row (sg_store_rows below: as they are, into rows of memory)
#pragma once
#include <cooperative_groups.h>

#include "common.cuh"
#include "umma.cuh"

#define SG_WORKERS 512
#define SG_WARPS (SG_WORKERS / 32)
#define SG_THREADS (SG_WORKERS + 64)
#define SG_PIECE 8                          // columns a warp stores at a time
#define SG_WAIT_LIMIT (1u << 24)

struct SgShared {
    unsigned long long full[2], empty[2], acc_full, acc_empty, rows_done, drained;
    unsigned tmem_base;
    int fail;                               // a wait ran out
};
__device__ __forceinline__ bool sg_wait(unsigned bar, unsigned parity, int* fail) {
    unsigned done = 0;
    for (unsigned it = 0; it < SG_WAIT_LIMIT; it++) {
        asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n" : "=r"(done) : "r"(bar), "r"(parity) : "memory");
        if (done) return true;
        if ((it & 255u) == 255u && *(volatile int*)fail) return false;
    }
    *(volatile int*)fail = 1;
    return false;
}
__device__ __forceinline__ bool sg_wait_warp(unsigned bar, unsigned parity, int* fail) { return __all_sync(0xffffffffu, sg_wait(bar, parity, fail)); }
// one arrival for the warp, after all of its lanes
__device__ __forceinline__ void sg_arrive(unsigned bar) {
    __syncwarp();
    if ((threadIdx.x & 31) == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// eight elements -> 16 bytes in each of the three planes
__device__ __forceinline__ void sg_cut(uint8_t* at, size_t plane, const float (&v)[8]) {
    unsigned h[4], m[4], l[4];
    auto nearest = [](float a, float b) {
        unsigned u;
        asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(u) : "f"(b), "f"(a));
        return u;
    };
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float a = v[2 * i], b = v[2 * i + 1];
        h[i] = nearest(a, b);
        const float a1 = a - __uint_as_float(h[i] << 16), b1 = b - __uint_as_float(h[i] & 0xffff0000u);
        m[i] = nearest(a1, b1);
        l[i] = nearest(a1 - __uint_as_float(m[i] << 16), b1 - __uint_as_float(m[i] & 0xffff0000u));
    }
    *(uint4*)at = make_uint4(h[0], h[1], h[2], h[3]);
    *(uint4*)(at + plane) = make_uint4(m[0], m[1], m[2], m[3]);
    *(uint4*)(at + 2 * plane) = make_uint4(l[0], l[1], l[2], l[3]);
}
__device__ __forceinline__ unsigned sg_offset(int row, int chunk) { return (unsigned)(row * 128 + ((chunk ^ (row & 7)) << 4)); }
// eight consecutive floats of a row of n, zeros behind its end
__device__ __forceinline__ void sg_load8(const float* p, int k, int n, bool vec, float (&v)[8]) {
    if (vec && k + 8 <= n) {
        const float4 x = *(const float4*)(p + k), y = *(const float4*)(p + k + 4);
        v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w; v[4] = y.x; v[5] = y.y; v[6] = y.z; v[7] = y.w;
    } else {
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = k + i < n ? p[k + i] : 0.0f;
    }
}
__device__ __forceinline__ void sg_zero8(float (&v)[8]) {
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = 0.0f;
}
__device__ __forceinline__ void sg_tmem16(unsigned addr, unsigned (&v)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]),
                   "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                 : "r"(addr));
}
// a warp's 32 rows x COUNT columns into rows of memory.  out: the row's first number (NULL: no such row); columns from `cols` on are dropped.  vec (rows start
// at multiples of 16 bytes): a thread stores its own row 16 bytes at a time -- eight stores and nothing else, where the way through shared memory, for rows
// that start anywhere, is a chain of some 500 instructions in two warps per scheduler (5000 cycles)
template <int COUNT>
__device__ __forceinline__ void sg_store_rows(float* buf, float* out, int cols, bool vec, const float (&v)[COUNT]) {
    if (vec) {
#pragma unroll
        for (int c = 0; c < COUNT; c += 4)
            if (out && c < cols) *(float4*)(out + c) = make_float4(v[c], v[c + 1], v[c + 2], v[c + 3]);
        return;
    }
    const int lane = threadIdx.x & 31;
    const unsigned long long at = (unsigned long long)out;
#pragma unroll
    for (int c0 = 0; c0 < COUNT; c0 += SG_PIECE) {
#pragma unroll
        for (int c = 0; c < SG_PIECE; c++) buf[lane * (SG_PIECE + 1) + c] = v[c0 + c];
        __syncwarp();
        const int c = c0 + lane % SG_PIECE;
#pragma unroll 4
        for (int r = lane / SG_PIECE; r < 32; r += 32 / SG_PIECE) {
            float* o = (float*)__shfl_sync(0xffffffffu, at, r);
            const float x = buf[r * (SG_PIECE + 1) + lane % SG_PIECE];
            if (o && c < cols) o[c] = x;
        }
        __syncwarp();
    }
}

__device__ __forceinline__ unsigned sg_runs(int steps, int half) { return steps ? (unsigned)(steps + half + 1) >> 1 : 0u; }

template <class P, bool SPLIT>
__global__ void __launch_bounds__(SG_THREADS, 1) split_gemm_kernel(const __grid_constant__ P p, int n_tiles, unsigned* err_dev, unsigned* err_host) {
    constexpr int N = 64 * P::HALVES, COUNT = N / 4;                  // COUNT: columns a warp collects
    constexpr unsigned A_PLANE = 128 * 128, B_PLANE = N * 128, A_BYTES = 3 * A_PLANE, B_BYTES = 3 * B_PLANE, STAGE = A_BYTES + B_BYTES;
    constexpr unsigned TMEM_COLS = P::HALVES == 1 ? 256 : 512;       // hh | hm + mh | hl + mm + lh
    constexpr unsigned TMA_BYTES = (P::A_TMA ? A_BYTES : 0) + B_BYTES;
    static_assert(!SPLIT || P::SHARED, "the other CTA's sums need the tiles' barriers");
    namespace cg = cooperative_groups;
    extern __shared__ __align__(1024) uint8_t sg_raw[];
    __shared__ SgShared sh;
    __shared__ typename P::Shared ps;
    uint8_t* ring = (uint8_t*)(((uintptr_t)sg_raw + 1023) & ~(uintptr_t)1023);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rank = SPLIT ? (int)cg::this_cluster().block_rank() : 0, first = SPLIT ? blockIdx.x >> 1 : blockIdx.x, stride = SPLIT ? gridDim.x >> 1 : gridDim.x;
    if (tid == 0) {
#pragma unroll
        for (int s = 0; s < 2; s++) { pg_mbar_init(pg_smem(&sh.full[s]), (P::A_TMA ? 0 : SG_WARPS) + 1); pg_mbar_init(pg_smem(&sh.empty[s]), 1); }
        pg_mbar_init(pg_smem(&sh.acc_full), 1); pg_mbar_init(pg_smem(&sh.acc_empty), SG_WARPS);
        pg_mbar_init(pg_smem(&sh.rows_done), SG_WARPS); pg_mbar_init(pg_smem(&sh.drained), 1);
        sh.fail = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == SG_WARPS) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(pg_smem(&sh.tmem_base)), "n"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    pg_fence_before();
    __syncthreads();
    pg_fence_after();
    const unsigned tmem = sh.tmem_base;
    pdl_enter();
    unsigned g = 0, runs = 0;                                         // steps and runs of the tiles before

    if (warp == SG_WARPS) {
        // ===== products: one thread =====
        for (int index = first; index < n_tiles; index += stride) {
            typename P::Tile tile;
            if (!p.tile(index, rank, tile)) continue;
            const int steps = tile.steps, half = tile.half;
            if (P::SHARED) {
                __syncthreads();
                if (*(volatile int*)&sh.fail) break;
                __syncthreads();
            }
            bool ok = true;
            if (lane == 0) {
                for (int s = 0; s < steps; s++) {
                    const unsigned gs = g + s, slot = gs & 1u, in_run = (s + half) >> 1;
                    const bool opens = s == 0 || !((s + half) & 1), closes = (s + half) & 1 || s + 1 == steps;
                    if (!(ok = sg_wait(pg_smem(&sh.full[slot]), (gs >> 1) & 1u, &sh.fail) && (!opens || sg_wait(pg_smem(&sh.acc_empty), ((runs + in_run) & 1u) ^ 1u, &sh.fail)))) break;
                    pg_fence_after();
                    const unsigned at = pg_smem(ring + (size_t)slot * STAGE);
                    const uint64_t ah = pg_smem_desc(at), am = pg_smem_desc(at + A_PLANE), al = pg_smem_desc(at + 2 * A_PLANE);
                    const uint64_t bh = pg_smem_desc(at + A_BYTES), bm = pg_smem_desc(at + A_BYTES + B_PLANE);
#pragma unroll
                    for (int kk = 0; kk < 4; kk++) {
                        const uint64_t adv = (uint64_t)((kk * PG_UMMA_K * 2) >> 4);
                        pg_umma_f16(tmem, ah + adv, bh + adv, pg_instr_desc(128, N, 1), !opens || kk > 0);                   // hh
                        pg_umma_f16(tmem + N, ah + adv, bm + adv, pg_instr_desc(128, 2 * N, 1), s > 0 || kk > 0);            //      hm | hl
                        pg_umma_f16(tmem + N, am + adv, bh + adv, pg_instr_desc(128, 2 * N, 1), 1u);                         //      mh | mm
                        pg_umma_f16(tmem + 2 * N, al + adv, bh + adv, pg_instr_desc(128, N, 1), 1u);                         //           lh
                    }
                    pg_umma_commit(pg_smem(&sh.empty[slot]));
                    if (closes) pg_umma_commit(pg_smem(&sh.acc_full));
                }
            }
            runs += sg_runs(steps, half);
            ok = __all_sync(0xffffffffu, ok);
            g += steps;
            if (SPLIT) {
                cg::this_cluster().sync();
                if (*(volatile int*)&sh.fail) break;
                cg::this_cluster().sync();
            }
            if (!ok) break;
        }
        if (lane == 0) {                                              // nothing of this CTA is in flight when its TMEM is given back
            int never = 0;
            pg_umma_commit(pg_smem(&sh.drained));
            sg_wait(pg_smem(&sh.drained), 0, &never);
        }
        __syncwarp();
    } else if (warp == SG_WARPS + 1) {
        // ===== TMA loads: one thread =====
        if (lane == 0) {
            if (P::A_TMA) asm volatile("prefetch.tensormap [%0];" ::"l"(p.map_a()) : "memory");
            asm volatile("prefetch.tensormap [%0];" ::"l"(p.map_b()) : "memory");
        }
        for (int index = first; index < n_tiles; index += stride) {
            typename P::Tile tile;
            if (!p.tile(index, rank, tile)) continue;
            if (P::SHARED) {
                __syncthreads();
                if (*(volatile int*)&sh.fail) break;
                __syncthreads();
            }
            bool ok = true;
            if (lane == 0) {
                for (int s = 0; s < tile.steps; s++) {
                    const unsigned gs = g + s, slot = gs & 1u, full = pg_smem(&sh.full[slot]), at = pg_smem(ring + (size_t)slot * STAGE);
                    if (!(ok = sg_wait(pg_smem(&sh.empty[slot]), ((gs >> 1) & 1u) ^ 1u, &sh.fail))) break;
                    pg_mbar_expect_tx(full, TMA_BYTES);
#pragma unroll
                    for (int i = 0; i < 3; i++) {
                        int x, y;
                        if (P::A_TMA) { p.at_a(tile, s, i, x, y); pg_tma_load_2d(at + i * A_PLANE, p.map_a(), full, x, y); }
                        p.at_b(tile, s, i, x, y);
                        pg_tma_load_2d(at + A_BYTES + i * B_PLANE, p.map_b(), full, x, y);
                    }
                }
            }
            ok = __all_sync(0xffffffffu, ok);
            g += tile.steps;
            if (SPLIT) {
                cg::this_cluster().sync();
                if (*(volatile int*)&sh.fail) break;
                cg::this_cluster().sync();
            }
            if (!ok) break;
        }
    } else {
        // ===== A, where it is cut here: elements 8 (tid / 128) .. and 32 later of the row tid % 128 =====
        const int ar0 = tid & 127, ac0 = tid >> 7;
        const int q = warp & 3, col0 = (warp >> 2) * COUNT, row = q * 32 + lane;         // collected: TMEM lanes 32 (warp % 4) .., COUNT columns
        const typename P::Fixed row_fixed = p.fixed(row), a_fixed = p.fixed(ar0);
        const unsigned a_at[2] = {sg_offset(ar0, ac0), sg_offset(ar0, ac0 + 4)};
        const unsigned from = tmem + ((unsigned)(q * 32) << 16) + (unsigned)col0;
        for (int index = first, nth = 0; index < n_tiles; index += stride) {
            typename P::Tile tile;
            if (!p.tile(index, rank, tile)) continue;
            const int steps = tile.steps, half = tile.half;
            if (P::SHARED) {
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");      // the sums that met in the stages, before TMA writes there again
                __syncthreads();
                if (*(volatile int*)&sh.fail) break;
                p.setup(tile, ps);
                __syncthreads();
            }
            typename P::ARow ar;
            float av[2][8], acc[COUNT];
            if (!P::A_TMA) {
                ar = p.a_row(tile, ps, a_fixed, ar0);
#pragma unroll
                for (int e = 0; e < 2; e++) if (steps > 0) p.load_a(tile, ar, 0, ac0 + 4 * e, av[e]);
            }
            bool ok = true;
#pragma unroll
            for (int c = 0; c < COUNT; c++) acc[c] = 0.0f;
            for (int s = 0; s <= steps; s++) {
                if (s < steps) {
                    const unsigned gs = g + s, slot = gs & 1u;
                    if (!P::A_TMA) {
                        if (!(ok = sg_wait_warp(pg_smem(&sh.empty[slot]), ((gs >> 1) & 1u) ^ 1u, &sh.fail))) break;
                        uint8_t* st = ring + slot * STAGE;
#pragma unroll
                        for (int e = 0; e < 2; e++) {
                            p.prep_a(tile, ar, av[e]);
                            sg_cut(st + a_at[e], A_PLANE, av[e]);
                            if (s + 1 < steps) p.load_a(tile, ar, s + 1, ac0 + 4 * e, av[e]);
                        }
                        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                        sg_arrive(pg_smem(&sh.full[slot]));
                    }
                } else if (P::SHARED) {
                    p.end_a(tile, ps, ar, ar0, ac0);
                    sg_arrive(pg_smem(&sh.rows_done));
                }
                if (s > 0 && (!((s + half) & 1) || s == steps)) {     // step s - 1 closed a run
                    if (!(ok = sg_wait_warp(pg_smem(&sh.acc_full), (runs + ((s - 1 + half) >> 1)) & 1u, &sh.fail))) break;
                    pg_fence_after();
#pragma unroll 1
                    for (int part = 0; part < (s < steps ? 1 : 3); part++) {
#pragma unroll
                        for (int c0 = 0; c0 < COUNT; c0 += 16) {
                            unsigned b[16];
                            sg_tmem16(from + part * N + c0, b);
                            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                            for (int c = 0; c < 16; c++) acc[c0 + c] += __uint_as_float(b[c]);
                        }
                    }
                    pg_fence_before();
                    sg_arrive(pg_smem(&sh.acc_empty));
                }
            }
            if (P::SHARED && ok) ok = sg_wait_warp(pg_smem(&sh.rows_done), (unsigned)nth & 1u, &sh.fail);
            bool nan = false;
#pragma unroll
            for (int c = 0; c < COUNT; c++) nan |= acc[c] != acc[c];
            if (nan && ok) {                                          // this CTA's share of the sum again, term by term
                const typename P::ARow a = p.a_row(tile, ps, row_fixed, row);
#pragma unroll 1
                for (int c = 0; c < COUNT; c++) {
                    const typename P::BCol b = p.b_col(tile, col0 + c);
                    float sum = 0.0f;
#pragma unroll 1
                    for (int k = 0; k < steps * 8; k++) {
                        float x[8], y[8];
                        typename P::ARow scratch = a;
                        p.load_a(tile, a, k >> 3, k & 7, x); p.prep_a(tile, scratch, x); p.load_b(tile, b, k >> 3, k & 7, y);
#pragma unroll
                        for (int i = 0; i < 8; i++) sum = P::SKIP_ZERO && x[i] == 0.0f ? sum : fmaf(x[i], y[i], sum);
                    }
#pragma unroll
                    for (int i = 0; i < COUNT; i++) acc[i] = i == c && acc[i] != acc[i] ? sum : acc[i];
                }
            }
            __syncwarp();
            float* buf = (float*)(ring + 2 * STAGE) + (size_t)warp * 32 * (SG_PIECE + 1);
            if (SPLIT) {
                cg::cluster_group cluster = cg::this_cluster();
                if (!ok) *(volatile int*)cluster.map_shared_rank(&sh.fail, rank ^ 1) = 1;      // neither goes on where the other gave up
                cluster.sync();                                       // both CTAs' stages are free
                if (*(volatile int*)&sh.fail) break;
                // columns of the lower half are finished by CTA 0, the others by CTA 1: each sends what the other needs
                const bool send = (warp >= SG_WARPS / 2) == (rank == 0);
                float4* sums = (float4*)ring + (size_t)(warp & (SG_WARPS / 2 - 1)) * (COUNT / 4) * 32 + lane;
                if (send) {
                    float4* to = cluster.map_shared_rank(sums, rank ^ 1);
#pragma unroll
                    for (int c = 0; c < COUNT; c += 4) to[c * 8] = make_float4(acc[c], acc[c + 1], acc[c + 2], acc[c + 3]);
                }
                p.give(ps, *cluster.map_shared_rank(&ps, rank ^ 1), tid);
                cluster.sync();
                if (!send) {
#pragma unroll
                    for (int c = 0; c < COUNT; c += 4) {
                        const float4 x = sums[c * 8];
                        acc[c] += x.x; acc[c + 1] += x.y; acc[c + 2] += x.z; acc[c + 3] += x.w;
                    }
                    p.emit(tile, ps, row_fixed, row, col0, acc, buf);
                }
            } else if (ok) p.emit(tile, ps, row_fixed, row, col0, acc, buf);
            if (!ok) break;
            g += steps; runs += sg_runs(steps, half); nth++;
        }
    }
    pg_fence_before();
    __syncthreads();
    if (warp == SG_WARPS) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(TMEM_COLS) : "memory");
    if (tid == 0 && sh.fail) {
        if (err_dev) atomicExch(err_dev, 5u);
        if (err_host) { *(volatile unsigned*)err_host = 5u; __threadfence_system(); }
    }
}

template <class P, bool SPLIT = false>
static int sg_launch(cc_device* dev, const P& p, int64_t n_tiles) {
    constexpr int smem = 2 * (3 * 128 * 128 + P::HALVES * 3 * 64 * 128) + 1024 + SG_WARPS * 32 * (SG_PIECE + 1) * 4;
    static_assert(smem + sizeof(typename P::Shared) + sizeof(SgShared) <= 227 * 1024, "one CTA's shared memory");
    CC_CUDA(dev, cudaFuncSetAttribute(split_gemm_kernel<P, SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    CC_REQUIRE(dev, n_tiles > 0 && n_tiles < ((int64_t)1 << 30), "split product: %lld tiles", (long long)n_tiles);
    int64_t at_once = SPLIT ? dev->sm_count / 2 : dev->sm_count;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2); cfg.blockDim = dim3(SG_THREADS); cfg.dynamicSmemBytes = smem; cfg.stream = dev->stream;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = SPLIT ? 2 : 1; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = dev->pdl ? 1 : 0;
    cfg.attrs = at;
    if (SPLIT) {                                                      // pairs that fit the chip at a time: an SM without a partner in its group stays idle
        cfg.numAttrs = 1;
        if (n_tiles > 64) {
            int pairs = 0;
            CC_CUDA(dev, cudaOccupancyMaxActiveClusters(&pairs, split_gemm_kernel<P, SPLIT>, &cfg));
            if (pairs > 0 && pairs < at_once) at_once = pairs;
        }
    }
    const unsigned ctas = (unsigned)(n_tiles < at_once ? n_tiles : at_once > 0 ? at_once : 1);
    cfg.gridDim = dim3(SPLIT ? 2 * ctas : ctas);
    cfg.numAttrs = 2;
    CC_CUDA(dev, cudaLaunchKernelEx(&cfg, split_gemm_kernel<P, SPLIT>, p, (int)n_tiles, dev->err_dev, dev->err_host));
    CC_LAUNCH_CHECK(dev);
    return CC_OK;
}
