// attn_rows.cuh -- attention of few query rows (decoding): scores, weights and values of a slice of the visible keys per CTA, and a second, short kernel that adds up
// the slices' results where there is more than one.  Included by seqops.cu behind WaGeom.
//
// A unit is one (query, key/value head, block of HB query heads, block of 1024 value columns).  Its visible keys are dealt out in equal contiguous slices; how
// many follows from the number of visible keys and the shapes (ar_slices), never from how many queries the call has.  A CTA takes its slice through shared
// memory by cp.async, a ring of tiles: key rows first, value rows behind them in the same ring, so that the values are on their way while the scores become
// weights; where a key row is also the value (latent attention) and the slice fits, it is read once.  A warp takes 4 keys x 8 heads of a tile, its lanes 4
// columns each, and passes its 32 sums on by halves; 4 value columns x 8 heads per lane behind that.  Up to 4 heads there is nothing to share: a warp reads its
// rows straight into registers (through the ring 16 heads of 128 over 4000 keys took 48 us, 2 barriers and 32 wavefronts of shared memory for 4 keys).
//
// A token, us, as a kernel of scores and one of values (the cache read once per 32 value columns) / here: 16 heads over 4000 latent rows (576, 512; 9.2 MB) 29 / 14.5, over
// 16000 72 / 38 ; 16 heads of their own (128) over 4000 keys (65 MB) 34 / 16, over 16000 113 / 51 ; 32 heads on 8 over 16000 (131 MB) 106 / 37 ; 128 heads (192, 128)
// over 4000 (655 MB) 240 / 130.  As a cluster of 8 CTAs a unit, the slices meeting in its shared memory and clusters through counters, the first took 21.5: 15 clusters are
// resident at a time (120 of 148 SMs), and the last cluster adds up what the others left.
//
// What bounds it: for few heads a key head the cache's bytes; for 16 heads over one latent row the reads of shared memory (12 of 16 bytes for 128 multiply-adds of
// a lane), and for short caches the chain launch, first load, sums.
#pragma once
#include "attn_rows_lanes.cuh"

#define AR_MACS (1 << 18)                // a slice has this many multiply-adds or AR_BYTES bytes, whichever are fewer keys, as long as there are SMs without one
#define AR_BYTES (1 << 17)
#define AR_WORKSPACE ((size_t)64 << 20)  // bytes of the slices' sums that a call has at a time
#define AR_LEAST 4                       // long caches: 4 slices at least, so that 64 sums or more of few terms are added up whatever the number of heads

struct ArArgs {
    const float *q, *k, *v, *r1, *r2, *sink;
    float *out, *part;                   // part: [unit][most][HB][dvp] sums of a slice
    float2* ml;                          // [unit][most][HB]: a slice's largest score and its sum of weights
    float scale;
    int most, cap, quantum, fine, late;  // slices of a unit: at most `most` in this call; by ar_slices
    int hblocks, cblocks, kv0;           // kv0: key/value head of the launch's first unit
    int dkp, dvp, rs, tile, stages, chunk, keep, vec, qvec;      // padded row lengths, floats; rs: floats of a ring row; keep: the ring holds the slice and its rows are the values
};
// how many slices n visible keys are dealt out in: `quantum` keys each; fewer than 8 of them leave the device far from full: twice as many, or `fine` keys each, up to 8;
// beyond 56 (5 queries of which fit the device at once) `late` keys each.  It never falls as n grows.
__host__ __device__ __forceinline__ int ar_parts(int n, int each) { return (int)(((unsigned)n + (unsigned)each - 1u) / (unsigned)each); }
__host__ __device__ __forceinline__ int ar_slices(int n, const ArArgs& A) {
    int c = ar_parts(n, A.quantum);
    if (c < 8) {
        c = c > 1 ? 2 * c : 1;
        if (A.fine != A.quantum) { const int f = ar_parts(n, A.fine); c = c > f ? c : f; }
        if (c > 8) c = 8;
    } else if (c > 56 && A.late != A.quantum) {
        const int l = ar_parts(n, A.late);
        c = l > 56 ? l : 56;
    }
    return c < A.cap ? c : A.cap;
}
__host__ __device__ constexpr int ar_stride(int HB) { return HB >= 8 ? HB + 4 : HB; }      // of a key's scores: whole float4, few bank conflicts down a head
__device__ __forceinline__ void ar_wait(int pending) {       // all but the newest `pending` groups of this thread's copies have arrived
    switch (pending) {
        case 0: asm volatile("cp.async.wait_group 0;" ::: "memory"); break;
        case 1: asm volatile("cp.async.wait_group 1;" ::: "memory"); break;
        case 2: asm volatile("cp.async.wait_group 2;" ::: "memory"); break;
        case 3: asm volatile("cp.async.wait_group 3;" ::: "memory"); break;
        case 4: asm volatile("cp.async.wait_group 4;" ::: "memory"); break;
        case 5: asm volatile("cp.async.wait_group 5;" ::: "memory"); break;
        default: asm volatile("cp.async.wait_group 6;" ::: "memory"); break;
    }
}
// one row of `cols` floats into shared memory by a warp, the tail up to a multiple of 4 zeros (cols 0: nothing but them)
__device__ __forceinline__ void ar_row(float* dst, const float* __restrict__ src, int cols, int vec, int lane) {
    const unsigned to = (unsigned)__cvta_generic_to_shared(dst);
    if (vec) {
        for (int c = lane * 4; c < cols; c += 128) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + c * 4), "l"(src + c) : "memory");
    } else {
        for (int c = lane; c < cols; c += 32) asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(to + c * 4), "l"(src + c) : "memory");
        if (lane < ((cols + 3) & ~3) - cols) dst[cols + lane] = 0.0f;
    }
}
// N sums spread over the lanes of a warp: lane l ends with the whole of sum l * N / 32
template <int N>
__device__ __forceinline__ float ar_fold(float (&v)[N], int lane) {
    int o = 16;
#pragma unroll
    for (int n = N / 2; n >= 1; n >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int i = 0; i < n; i++) {
            const float give = up ? v[i] : v[i + n], mine = up ? v[i + n] : v[i];
            v[i] = mine + __shfl_xor_sync(0xffffffffu, give, o);
        }
        o >>= 1;
    }
    float s = v[0];
    for (; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}
__device__ __forceinline__ void ar_fma4(float4& a, float p, const float4& v) { a.x = fmaf(p, v.x, a.x); a.y = fmaf(p, v.y, a.y); a.z = fmaf(p, v.z, a.z); a.w = fmaf(p, v.w, a.w); }

// a row's 4 columns from c on, zeros behind its end
__device__ __forceinline__ float4 ar_load4(const float* __restrict__ row, int c, int cols, int vec) {
    if (vec) return __ldg((const float4*)(row + c));
    return make_float4(row[c], c + 1 < cols ? row[c + 1] : 0.0f, c + 2 < cols ? row[c + 2] : 0.0f, c + 3 < cols ? row[c + 3] : 0.0f);
}
// grid (slices, queries, units of a query)
template <int HB>
__global__ void __launch_bounds__(AR_THREADS, HB <= 4 ? 2 : 1) attn_rows_kernel(ArArgs A, WaGeom g) {
    constexpr bool DIRECT = HB <= 4;
    extern __shared__ __align__(16) float ar_sm[];
    constexpr int HS = HB < 8 ? HB : 8, HG = HB / HS, PS = ar_stride(HB), KU = 4, EARLY = 4;
    __shared__ float top[HB], sum[HB], fac[HB];
    float* qs = ar_sm;                                             // [HB][dkp]
    float* sc = qs + HB * A.dkp;                                   // [chunk][PS]
    float* ring = sc + (size_t)A.chunk * PS;                       // [stages][tile][rs]; behind the last tile the warps' sums [key group][HB][dvp]
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned kcb = blockIdx.z / (unsigned)A.cblocks, ukv = kcb / (unsigned)A.hblocks;
    const int slice = blockIdx.x, t = blockIdx.y, cb = (int)(blockIdx.z - kcb * A.cblocks), hb = (int)(kcb - ukv * A.hblocks), kvh = A.kv0 + (int)ukv;
    const int h0 = kvh * g.R + hb * HB, nh = min(HB, g.R - hb * HB), c_first = cb * AR_COLS, cols = ar_cols(g.dv, cb);
    const int64_t i = g.pos0 + t, lo = wa_lo(g, i);
    const int n = (int)(i - lo) + 1, slices = ar_slices(n, A);     // n: at most the ring's rows
    const int per = (int)((unsigned)(n + slices - 1) / (unsigned)slices), s0 = min(n, slice * per), m = min(n - s0, per);
    const float* kbase = A.k + (int64_t)kvh * g.dk;
    const float* vbase = A.v + (int64_t)kvh * g.vhs + c_first;
    const float* qrow = A.q + ((int64_t)t * g.H + h0) * g.dk;
    const ArLane at_v = ar_lane(w, lane, A.dvp, cols, HG);
    const int kgs = at_v.kgs, hg = at_v.hg, kg = at_v.kg, col = at_v.col;
    const bool loads = at_v.loads;
    pdl_enter();                                                   // up to here nothing but the arguments
    if (slice >= slices) return;
    float4 acc[HS];
#pragma unroll
    for (int h = 0; h < HS; h++) acc[h] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    int c0 = 0;
    do {                                                           // chunks of a slice (one but for the longest caches; an empty slice: once)
        const int mc = min(A.chunk, m - c0);
        const int nk = DIRECT ? 0 : (mc + A.tile - 1) / A.tile, nt = DIRECT ? 0 : A.keep ? nk : 2 * nk;
        const int64_t p0 = lo + s0 + c0, r0 = p0 >> 31 ? p0 % g.ring : (int64_t)((unsigned)p0 % (unsigned)g.ring);
        auto load = [&](int j) {                                   // tile j of the chunk: nk of keys, nk of values
            const bool val = j >= nk;
            const int at = (val ? j - nk : j) * A.tile, rows = min(A.tile, mc - at);
            float* dst = ring + (size_t)(j % A.stages) * A.tile * A.rs;
            for (int r = w; r < rows; r += AR_WARPS) {
                int64_t row = r0 + at + r;
                if (row >= g.ring) row -= g.ring;
                if (val) ar_row(dst + (size_t)r * A.rs, vbase + row * g.vrs, cols, A.vec, lane);
                else ar_row(dst + (size_t)r * A.rs, kbase + row * g.krs, g.dk, A.vec, lane);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        int issued = 0;
        if (c0 == 0)                                               // the queries come with the first tile
            for (int h = w; h < HB; h += AR_WARPS) {
                if (h < nh) ar_row(qs + h * A.dkp, qrow + (int64_t)h * g.dk, g.dk, A.qvec, lane);
                else
                    for (int d = lane; d < A.dkp; d += 32) qs[h * A.dkp + d] = 0.0f;
            }
        const int ahead = A.keep ? A.stages : A.stages - 1;
        while (issued < min(nt, ahead)) load(issued++);
        auto score = [&](float s, int c, int h) {                  // score of key c of the chunk, head h of the block
            s *= A.scale;
            if (g.softcap > 0.0f) s = g.softcap * tanhf(s / g.softcap);
            if (A.r1 && h < nh) s -= A.r1[h0 + h] * log1pf(A.r2[h0 + h] * (float)(i - (lo + s0 + c0 + c)));
            sc[c * PS + h] = s;
        };
        auto value4 = [&](int c) {                                 // 4 columns of value row c of the chunk
            int64_t row = r0 + c;
            if (row >= g.ring) row -= g.ring;
            return ar_load4(vbase + row * g.vrs, col, cols, A.vec);
        };
        // KU keys x HS heads, rows from shared memory or not
        auto unit = [&](auto key4, auto q4, int c, int rows, int h) {
            float s[KU * HS];
#pragma unroll
            for (int x = 0; x < KU * HS; x++) s[x] = 0.0f;
#pragma unroll 1
            for (int d = lane * 4; d < A.dkp; d += 128) {
                float4 kv[KU];
#pragma unroll
                for (int r = 0; r < KU; r++) kv[r] = key4(r, d);
#pragma unroll
                for (int x = 0; x < HS; x++) {
                    const float4 qv = q4(x, d);
#pragma unroll
                    for (int r = 0; r < KU; r++) {
                        float y = s[r * HS + x];
                        y = fmaf(qv.x, kv[r].x, y); y = fmaf(qv.y, kv[r].y, y); y = fmaf(qv.z, kv[r].z, y); y = fmaf(qv.w, kv[r].w, y);
                        s[r * HS + x] = y;
                    }
                }
            }
            const float r = ar_fold<KU * HS>(s, lane);
            const int id = lane * (KU * HS) / 32;
            if (lane % (32 / (KU * HS)) == 0 && id / HS < rows) score(r, c + id / HS, h + id % HS);
        };
        if constexpr (DIRECT) {
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();
            for (int c = w * KU; c < mc; c += AR_WARPS * KU) {
                const float* kr[KU];
#pragma unroll
                for (int r = 0; r < KU; r++) {
                    int64_t row = r0 + min(c + r, mc - 1);
                    if (row >= g.ring) row -= g.ring;
                    kr[r] = kbase + row * g.krs;
                }
                unit([&](int r, int d) { return ar_load4(kr[r], d, g.dk, A.vec); }, [&](int x, int d) { return *(const float4*)(qs + x * A.dkp + d); }, c, mc - c, 0);
            }
        } else {
            for (int j = 0; j < nk; j++) {
                ar_wait(issued - j - 1);
                __syncthreads();
                if (issued < nt) load(issued++);
                const float* kt = ring + (size_t)(j % A.stages) * A.tile * A.rs;
                const int at = j * A.tile, rows = min(A.tile, mc - at);
                for (int u = w; u < (rows + 3) / 4 * HG; u += AR_WARPS) {
                    const int c = u / HG * 4, h = u % HG * HS;
                    const float* kr = kt + (size_t)c * A.rs;
                    const float* qr = qs + h * A.dkp;
                    unit([&](int r, int d) { return *(const float4*)(kr + r * A.rs + d); }, [&](int x, int d) { return *(const float4*)(qr + x * A.dkp + d); }, at + c, rows - c, h);
                }
            }
        }
        float4 early[EARLY];                                       // a warp's first value rows come while the scores become weights (4 heads: no registers for it)
        if constexpr (HB <= 2) {
#pragma unroll
            for (int x = 0; x < EARLY; x++)
                if (loads && kg + x * kgs < mc) early[x] = value4(kg + x * kgs);
        }
        __syncthreads();
        for (int h = w; h < HB; h += AR_WARPS) {                   // scores -> weights relative to the largest so far; none where there is no score but -inf
            const float before = c0 ? top[h] : -INFINITY;
            float mx = before;
            for (int c = lane; c < mc; c += 32) mx = fmaxf(mx, sc[c * PS + h]);
            mx = warp_max(mx);
            float tot = 0.0f;
            for (int c = lane; c < mc; c += 32) {
                const float s = sc[c * PS + h], e = s == -INFINITY ? 0.0f : expf(s - mx);
                sc[c * PS + h] = e;
                tot += e;
            }
            tot = warp_sum(tot);
            __syncwarp();
            if (lane == 0) {
                const float f = before == -INFINITY ? 0.0f : expf(before - mx);
                fac[h] = f; top[h] = mx; sum[h] = c0 ? fmaf(f, sum[h], tot) : tot;
            }
        }
        __syncthreads();
        if (c0) {
#pragma unroll
            for (int h = 0; h < HS; h++) {
                const float f = fac[hg * HS + h];
                acc[h].x *= f; acc[h].y *= f; acc[h].z *= f; acc[h].w *= f;
            }
        }
        auto add = [&](const float4& v, const float* p) {          // a value row's 4 columns, weighted for each head
            if constexpr (HS >= 4) {
#pragma unroll
                for (int h = 0; h < HS; h += 4) {
                    const float4 e = *(const float4*)(p + h);
                    ar_fma4(acc[h], e.x, v); ar_fma4(acc[h + 1], e.y, v); ar_fma4(acc[h + 2], e.z, v); ar_fma4(acc[h + 3], e.w, v);
                }
            } else {
#pragma unroll
                for (int h = 0; h < HS; h++) ar_fma4(acc[h], p[h], v);
            }
        };
        if constexpr (DIRECT) {
            if (loads) {
                int c = kg;
                if constexpr (HB <= 2) {
#pragma unroll
                    for (int x = 0; x < EARLY; x++)
                        if (kg + x * kgs < mc) add(early[x], sc + (kg + x * kgs) * PS);
                    c += EARLY * kgs;
                }
#pragma unroll 4
                for (; c < mc; c += kgs) add(value4(c), sc + c * PS);
            }
        } else {
            for (int j = 0; j < nk; j++) {
                if (!A.keep) {
                    ar_wait(issued - (nk + j) - 1);
                    __syncthreads();
                    if (issued < nt) load(issued++);
                }
                const float* vt = ring + (size_t)((A.keep ? j : nk + j) % A.stages) * A.tile * A.rs;
                const int at = j * A.tile, rows = min(A.tile, mc - at);
                if (loads) {
#pragma unroll 4
                    for (int c = kg; c < rows; c += kgs) add(*(const float4*)(vt + (size_t)c * A.rs + col), sc + (at + c) * PS + hg * HS);
                }
            }
        }
        c0 += A.chunk;
        __syncthreads();                                           // ring and weights have been read
    } while (c0 < m);

    // the warps' sums, in the order of the key groups
    const int row4 = A.dvp / 4, items = HB * row4;             // float4 numbers
    float4* red = (float4*)ring;
    if (at_v.sums) {
#pragma unroll
        for (int h = 0; h < HS; h++) red[kg * items + (hg * HS + h) * row4 + col / 4] = acc[h];
    }
    __syncthreads();
    const size_t at = ((size_t)t * gridDim.z + blockIdx.z) * A.most + slice;
    if (slices > 1) {
        for (int e = threadIdx.x; e < items; e += AR_THREADS) {
            float4 a = red[e];
            for (int x = 1; x < kgs; x++) { const float4 b = red[x * items + e]; a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w; }
            ((float4*)A.part)[at * items + e] = a;
        }
        if (threadIdx.x < HB) A.ml[at * HB + threadIdx.x] = make_float2(top[threadIdx.x], sum[threadIdx.x]);
        return;
    }
    for (int e = threadIdx.x; e < HB * A.dvp; e += AR_THREADS) {
        float a = ((const float*)red)[e];
        for (int x = 1; x < kgs; x++) a += ((const float*)red)[x * HB * A.dvp + e];
        const int h = e / A.dvp, c = e - h * A.dvp;
        if (h >= nh || c >= cols) continue;
        // a sink is one more slice: a sum of weights 1 and no value
        const float sk = A.sink ? A.sink[h0 + h] : -INFINITY, mx = fmaxf(sk, top[h]), f = top[h] == -INFINITY ? 0.0f : expf(top[h] - mx);
        A.out[((int64_t)t * g.H + h0 + h) * g.dv + c_first + c] = a * f / (f * sum[h] + (sk == -INFINITY ? 0.0f : expf(sk - mx)));
    }
}
// the slices of a unit added up: grid (items / 8, queries, units of a query), an item is 4 columns of a head.  64 groups of 8 threads take every 64th slice, all of
// their loads at once, and their parts are added up by halves of the warp, then warp by warp, the sink behind them.
#define AR_GROUPS (AR_THREADS / 8)
#define AR_EACH 5
__global__ void __launch_bounds__(AR_THREADS) attn_rows_sum_kernel(ArArgs A, WaGeom g, int HB) {
    __shared__ float4 sa[AR_WARPS][8];
    __shared__ float sm[AR_WARPS][8], st[AR_WARPS][8];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, row4 = A.dvp / 4, items = HB * row4, x = lane & 7, z0 = threadIdx.x >> 3;
    const unsigned kcb = blockIdx.z / (unsigned)A.cblocks, ukv = kcb / (unsigned)A.hblocks;
    const int t = blockIdx.y, cb = (int)(blockIdx.z - kcb * A.cblocks), hb = (int)(kcb - ukv * A.hblocks), kvh = A.kv0 + (int)ukv;
    const int64_t i = g.pos0 + t;
    const int n = (int)(i - wa_lo(g, i)) + 1, slices = ar_slices(n, A);
    pdl_enter();                                                   // up to here nothing but the arguments
    if (slices <= 1) return;
    const int e = min((int)blockIdx.x * 8 + x, items - 1), h = e / row4;
    const size_t unit = ((size_t)t * gridDim.z + blockIdx.z) * A.most;
    float2 p[AR_EACH];
    float4 v[AR_EACH];
    float mx = -INFINITY;
#pragma unroll
    for (int y = 0; y < AR_EACH; y++) {
        const int z = z0 + y * AR_GROUPS;
        p[y] = make_float2(-INFINITY, 0.0f); v[y] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (z < slices) { p[y] = A.ml[(unit + z) * HB + h]; v[y] = ((const float4*)A.part)[(unit + z) * items + e]; }
    }
#pragma unroll
    for (int y = 0; y < AR_EACH; y++) mx = fmaxf(mx, p[y].x);
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8)); mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
    if (lane < 8) sm[w][x] = mx;
    const int head = kvh * g.R + hb * HB + h;
    const bool in = (int)blockIdx.x * 8 + x < items && hb * HB + h < g.R;
    const float sk = A.sink && in ? A.sink[head] : -INFINITY;
    __syncthreads();
    mx = sk;
#pragma unroll
    for (int y = 0; y < AR_WARPS; y++) mx = fmaxf(mx, sm[y][x]);
    float4 a = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    float tot = 0.0f;
#pragma unroll
    for (int y = 0; y < AR_EACH; y++) {
        const float f = p[y].x == -INFINITY ? 0.0f : expf(p[y].x - mx);
        tot = fmaf(f, p[y].y, tot);
        ar_fma4(a, f, v[y]);
    }
#pragma unroll
    for (int o = 8; o < 32; o *= 2) {
        a.x += __shfl_xor_sync(0xffffffffu, a.x, o); a.y += __shfl_xor_sync(0xffffffffu, a.y, o);
        a.z += __shfl_xor_sync(0xffffffffu, a.z, o); a.w += __shfl_xor_sync(0xffffffffu, a.w, o);
        tot += __shfl_xor_sync(0xffffffffu, tot, o);
    }
    if (lane < 8) { sa[w][x] = a; st[w][x] = tot; }
    __syncthreads();
    if (threadIdx.x >= 32) return;
    // a column a thread
    const float* col = (const float*)&sa[0][0] + lane;
    const int from = lane >> 2, c = (lane & 3);
    float sum = col[0], div = st[0][from];
#pragma unroll
    for (int y = 1; y < AR_WARPS; y++) { sum += col[y * 32]; div += st[y][from]; }
    const int e1 = min((int)blockIdx.x * 8 + from, items - 1), h1 = e1 / row4, at = cb * AR_COLS + (e1 - h1 * row4) * 4 + c, head1 = kvh * g.R + hb * HB + h1;
    if ((int)blockIdx.x * 8 + from >= items || hb * HB + h1 >= g.R || at >= g.dv) return;
    const float sk1 = A.sink ? A.sink[head1] : -INFINITY;
    float mx1 = sk1;
#pragma unroll
    for (int y = 0; y < AR_WARPS; y++) mx1 = fmaxf(mx1, sm[y][from]);
    if (sk1 != -INFINITY) div += expf(sk1 - mx1);
    A.out[((int64_t)t * g.H + head1) * g.dv + at] = sum / div;
}

template <int HB>
static int ar_launch(cc_device* dev, const ArArgs& A, const WaGeom& g, size_t smem) {
    const unsigned units = (unsigned)(g.G * A.hblocks * A.cblocks);
    if (smem > 40 * 1024) CC_CUDA(dev, cudaFuncSetAttribute(attn_rows_kernel<HB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    cc_launch_pdl(dev, attn_rows_kernel<HB>, dim3((unsigned)A.most, (unsigned)g.T, units), AR_THREADS, smem, A, g);
    if (A.most > 1) {
        dev->launches++;
        cc_launch_pdl(dev, attn_rows_sum_kernel, dim3((unsigned)(HB * A.dvp / 4 + 7) / 8, (unsigned)g.T, units), AR_THREADS, 0, A, g, HB);
    }
    CC_LAUNCH_CHECK(dev);
    return CC_OK;
}
// A filled with the operands; reach: the most keys one query sees
static int attn_rows(cc_device* dev, const WaGeom& g, ArArgs A, int reach) {
    const size_t most = 200 * 1024;
    const bool lat = A.v == A.k && g.vrs == g.krs;
    A.dkp = (g.dk + 3) & ~3;
    A.cblocks = (g.dv + AR_COLS - 1) / AR_COLS;
    A.dvp = ar_dvp(g.dv);
    A.vec = g.dk % 4 == 0 && g.krs % 4 == 0 && g.vrs % 4 == 0 && g.vhs % 4 == 0 && g.dv % 4 == 0 && (((uintptr_t)A.k | (uintptr_t)A.v) & 15) == 0;
    A.qvec = g.dk % 4 == 0 && ((uintptr_t)A.q & 15) == 0;
    int HB = g.R > 8 ? 16 : g.R > 4 ? 8 : g.R > 2 ? 4 : g.R;
    while (HB > 1 && (size_t)HB * A.dkp * 4 > 72 * 1024) HB /= 2;
    size_t smem = 0;
    for (;; HB /= 2) {
        A.hblocks = (g.R + HB - 1) / HB;
        const int64_t per_query = (int64_t)g.G * A.hblocks * A.cblocks, sms = HB <= 4 ? 2 * dev->sm_count : dev->sm_count;      // up to 4 heads two CTAs fit an SM
        const int64_t cap = sms / per_query, cols = g.dk + g.dv / A.cblocks, by_macs = AR_MACS / (HB * cols), by_bytes = AR_BYTES / (4 * cols);
        A.cap = (int)(cap < AR_LEAST ? AR_LEAST : cap < AR_GROUPS * AR_EACH ? cap : AR_GROUPS * AR_EACH);
        A.quantum = (int)(by_macs < by_bytes ? by_macs : by_bytes);
        A.quantum = A.quantum < 8 ? 8 : A.quantum;
        // through the ring of tiles a slice of many narrow rows takes longer than the kernel that adds up several.  us as one slice / in up to 8: 8 heads a key head (2 of 64) over 200
        // keys 18.0 / 10.2, over 500 14.6 / 10.3 (2 / 8 slices) ; 16 heads a key head (2 of 64) over 100 16.1 / 9.5.  Up to 4 heads a second kernel costs more: 200 keys of 64 9.3 / 10.0
        A.fine = HB > 4 && A.quantum > 512 / HB ? 512 / HB : A.quantum;
        // few heads over wide rows: a CTA of 30 rows is short, and several queries are more of them than fit the device at once.  2300 latent rows, us by 30 / by 45 keys: 1 head, 1 query
        // 12.6 / 12.7, 4 queries 19.2 / 13.6, 5 20.4 / 13.6, 6 21.3 / 20.8, 12 34 / 29.5, 25 59 / 51 ; 4 heads, 2 queries 15.8 / 16.8, 5 26.5 / 19.2, 6 27.4 / 28.8, 12 47 / 42
        A.late = HB <= 4 && cols > 512 ? A.quantum * 3 / 2 : A.quantum;
        A.most = ar_slices(reach, A);
        // the longest slice of a row that sees up to `reach` keys
        const int last = (reach + A.most - 1) / A.most, slice = A.most > 1 && A.late > last ? A.late : last;      // (a row of fewer keys: no more than `late` a slice)
        const int chunk_most = HB == 16 ? 512 : HB == 8 ? 1024 : 2048 / HB;
        A.chunk = slice < chunk_most ? (slice + 3) & ~3 : chunk_most;
        const size_t fixed = ((size_t)HB * A.dkp + (size_t)A.chunk * ar_stride(HB)) * 4, sums = (size_t)AR_WARPS * (HB < 8 ? HB : 8) * 128 * 4;
        size_t ring = 0;
        A.stages = 1;
        if (HB > 4) {
            A.rs = lat && A.cblocks == 1 ? A.dkp : A.dkp > A.dvp ? A.dkp : A.dvp;
            // a tile is 4 keys a warp (a pair of warps with 8 heads each), less where that is more than 36 KB; the slice as a whole where its rows are the values and it fits
            const size_t row = (size_t)A.rs * 4, whole = ((slice + 3) & ~3) * row;
            A.keep = lat && A.cblocks == 1 && A.chunk >= slice && fixed + whole <= most;
            A.stages = A.keep ? 1 : 4;
            A.tile = A.keep ? (slice + 3) & ~3 : HB == 16 ? 32 : 64;
            if (!A.keep)
                while (A.tile > 4 && (A.tile * row > 36 * 1024 || fixed + A.stages * A.tile * row > most)) A.tile /= 2;
            ring = A.stages * A.tile * row;
        }
        smem = fixed + (ring > sums ? ring : sums);
        if (HB <= 4 || smem <= most) break;
    }
    // short caches: a CTA a head.  The slices, and with them the order of every sum, stay those of the larger block
    if (HB <= 4 && A.chunk < 512 && (int64_t)g.T * g.G * A.hblocks * HB * A.most <= 2 * dev->sm_count) {
        HB = 1; A.hblocks = g.R;
        smem = (size_t)(A.dkp + A.chunk + AR_WARPS * 128) * 4;
    }
    // queries in portions whose partial sums take AR_WORKSPACE at most (many of them come here where tiles have no room), key heads in as many as a grid has units.  A query's
    // slices, and its bits, are the same in any portion
    const int64_t blocks = (int64_t)A.hblocks * A.cblocks, fit = 65535 / blocks > 0 ? 65535 / blocks : 1, heads = g.G < fit ? g.G : fit;
    const size_t part = (size_t)(heads * blocks) * A.most * HB * A.dvp * 4, ml = (size_t)(heads * blocks) * A.most * HB * 8;      // of one query
    const int64_t room = A.most > 1 && AR_WORKSPACE / (part + ml) < (size_t)g.T ? (int64_t)(AR_WORKSPACE / (part + ml)) : g.T, portion = room > 0 ? room : 1;
    void* ws = nullptr; size_t cls = 0;
    if (A.most > 1) {
        int rc = cc_pool_alloc(dev, (size_t)portion * (part + ml), &ws, &cls);
        if (rc) return rc;
        A.part = (float*)ws; A.ml = (float2*)((uint8_t*)ws + portion * part);
    }
    int rc = CC_OK;
    for (int64_t t0 = 0; t0 < g.T && rc == CC_OK; t0 += portion)
        for (int64_t kv0 = 0; kv0 < g.G && rc == CC_OK; kv0 += heads) {
            ArArgs B = A;
            WaGeom p = g;
            B.q += t0 * g.H * g.dk; B.out += t0 * g.H * g.dv; B.kv0 = (int)kv0;
            p.pos0 += t0; p.T = (int)(g.T - t0 < portion ? g.T - t0 : portion); p.G = (int)(g.G - kv0 < heads ? g.G - kv0 : heads);
            rc = HB == 16 ? ar_launch<16>(dev, B, p, smem) : HB == 8 ? ar_launch<8>(dev, B, p, smem) : HB == 4 ? ar_launch<4>(dev, B, p, smem)
                 : HB == 2 ? ar_launch<2>(dev, B, p, smem) : ar_launch<1>(dev, B, p, smem);
        }
    if (ws) cc_pool_free(dev, ws, cls);
    return rc;
}
