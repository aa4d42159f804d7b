// mega_ring.cu -- the persistent decode kernel with the weight stream decoupled from the compute warps.
//
// Why (profiles/r02d, r02g): in mega.cu every warp alternates "issue the loads of a segment" and "consume a segment"; at a phase
// boundary (slowest warp -> grid barrier -> activation prologue, 6-9 us) no warp issues loads, so only the 2 look-ahead segments per
// warp (20 MB per GPU, 3 us of HBM time) cover the bubble and HBM idles for the rest: 2.36 ms per Llama-2-7B Q8_0 token against
// 1.07 ms of pure streaming.  Weights are immutable, so nothing forces the weight stream to follow the phase order of the compute:
//   * warps 16-18 of every CTA are PRODUCERS: their threads walk the phase table on their own, ahead of the compute warps, and issue cp.async.bulk (TMA) copies
//     of items -- two rows' segment of 128 blocks: 8192 B of Q8_0 quants + 512 B of f16 scales (1024 B are theirs) -- into a ring of shared-memory slots, as many as fit beside
//     the per-phase working area (17 to 19 = 160-174 KB per SM, 25 MB per GPU).  They never wait for a barrier or an activation: whenever a slot is free the
//     next item of this CTA's rows -- of this phase or any later one -- is being fetched.
//   * warp 19 asks L2 for the items behind the ring: it is ahead of the copies by a ring's size and 224 KB (390 KB per SM, 58 MB per GPU) at most, at 20 B per cycle and
//     SM: a full ring is 4 us of HBM time, the time between one phase's last row and the next one's first 5 to 7 us, the attention phase 7.  A 7B Q8_0 token 1862 ->
//     1814 us (with 120 KB instead of the 224 1830; 224 and 300 KB, 20 and 26 B alike; 417 KB, 86 MB per GPU with the ring's size, was 30 % slower: more than L2 keeps).
//     Lead and pace count every item as a full one: items of rows of 288 are charged 14 times their bytes, the copies overtake the requests, and short rows come by the
//     ring alone.  Without a pace the requests queue in front of the barrier's own traffic: with 19 MB under way a barrier takes 20 us instead of 2 (measured by
//     itself; at 6.3 TB/s with 7 MB under way 3.4).
//   * warps 0-15 are CONSUMERS: the CTA's rows are one contiguous run, two neighbouring rows an item, a warp each; same per-lane block order, same arithmetic as
//     mega.cu / matvec_stream.cu (bit-identical results), but a segment is read from the ring with LDS.128 after waiting on the slot's "full" mbarrier, and
//     the slot is handed back through its "done" words.  The activation stays in registers, lanes' sums are added up behind the row loop.  (One warp on both
//     rows of an item, activation from shared memory: 16 of the 19 slots were being read and only the others under way, 1950 us a token; now 1814.)
//     96 registers a thread are enough, and next to nothing may spill (4 bytes do, 84 where the K-quant phases are compiled in): a spilled register is a trip to L2,
//     the ring leaves no L1 (the same rows with a prologue that kept its row in registers, 600 bytes of spills: 2540 us).
// The 512 compute threads synchronise on named barrier 1 (MK_SYNC); the producer warps never join it.
// 20 warps: five per SM sub-partition, so its 16384 registers allow 96 per thread (what __launch_bounds__(640, 1) yields).
#define MK_SYNC() asm volatile("bar.sync 1, 512;" ::: "memory")
#define MK_GENERIC_NOINLINE 1
#include "mega_phases.cuh"
#include "quotients.cuh"

#define MR_PRODUCER_WARPS 4        // 20 warps: five per SM sub-partition, still 96 registers per thread
#define MR_ISSUERS 96                // threads that issue copies: three warps (two: +1 %); the fourth warp prefetches
#define MR_L2_LEAD (224 * 1024)       // bytes of items, beside a ring's size, that the requests to L2 are ahead of the copies, per SM
#define MR_L2_RATE 20                 // bytes per cycle and SM at which they are asked for: 5.8 TB/s
#define MR_THREADS (MK_THREADS + 32 * MR_PRODUCER_WARPS)
#define MR_MAX_SLOTS 56
#define MR_DESC_WORDS ((int)(sizeof(MkPhase) / 4))
#define MR_DESC_PER_LANE ((MR_DESC_WORDS + 31) / 32)

struct MrRing {
    int ring_off;          // byte offset of the ring in dynamic shared memory (16-byte aligned)
    int slot_bytes;        // bytes per slot (multiple of 128): quants of up to 4 groups, then their f16 scales
    int nslots;
    int at_ch;             // ATTN phase: cache rows per TMA chunk
};

__device__ __forceinline__ void mr_expect_tx(unsigned bar, unsigned bytes) { asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory"); }
__device__ __forceinline__ void mr_bulk_g2s(unsigned dst, const void* src, unsigned bytes, unsigned bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ bool mr_try_wait(unsigned bar, unsigned parity) {
    unsigned ok;
    asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// Slot hand-back: the consumer stores (item number + 1) into the slot's "done" word (release), the producer polls it (acquire) for
// exactly the previous tenant's number -- an mbarrier parity could not tell one lap from two.  `dep` ties the store behind the
// arithmetic that consumed the slot's data.
__device__ __forceinline__ void mr_release(unsigned done_addr, unsigned v, float dep) { asm volatile("st.release.cta.shared::cta.u32 [%0], %1;" ::"r"(done_addr), "r"(v), "f"(dep) : "memory"); }
__device__ __forceinline__ unsigned mr_ld_acquire_shared(unsigned addr) {
    unsigned v;
    asm volatile("ld.acquire.cta.shared::cta.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}

// Rows of a streaming MATVEC phase that belong to this CTA: one contiguous run.  They go through the ring as ITEMS: one segment of a GROUP, two rows next to each
// other in one matrix (gate and up rows of two units are two groups, one behind the other).  Where a segment is a whole row the two lie in one run: two copies
// an item, quants and scales -- the copy engine takes 30 M requests/s and SM, and a gate row beside an up row, four copies an item, was bound by that (10.3 us of
// 75 items).  Producer and consumers derive the same item sequence from this: group P, segment s = item P * NSEG + s.
struct MrGeo {
    int nb, GR, NSEG, n_rows, groups, first, last_half_off;
    bool pair;
};
__device__ __forceinline__ MrGeo mr_geo(const StreamArgs& A) {
    MrGeo g;
    g.nb = A.k >> 5; g.GR = (g.nb + 31) >> 5; g.NSEG = (g.GR + MK_SEG - 1) / MK_SEG;
    g.pair = A.epilogue == 2;
    const StreamMats& M = A.mats;
    const int m_cat = g.pair ? M.m[0] : M.m[0] + (M.n > 1 ? M.m[1] : 0) + (M.n > 2 ? M.m[2] : 0);
    if (A.epilogue == 3) {             // exchange phases: blocks of a multiple of 4 rows (mega.cu mk_geo)
        const int rpc = (((m_cat + (int)gridDim.x - 1) / (int)gridDim.x) + 3) & ~3;
        g.first = (int)blockIdx.x * rpc;
        g.n_rows = min(rpc, max(0, m_cat - g.first));
    } else {
        const int each = m_cat / (int)gridDim.x, more = m_cat - each * (int)gridDim.x;
        g.first = (int)blockIdx.x * each + min((int)blockIdx.x, more);
        g.n_rows = each + ((int)blockIdx.x < more ? 1 : 0);
    }
    g.groups = ((g.n_rows + 1) >> 1) << (g.pair ? 1 : 0);
    g.last_half_off = 16 * (g.nb - 32 * (g.GR - 1));
    return g;
}
// first row of a group, counted from the CTA's first
__device__ __forceinline__ int mr_unit(const MrGeo& g, int P) { return g.pair ? P & ~1 : 2 * P; }
// concatenated row -> (matrix, row of it)
__device__ __forceinline__ int mr_locate(const StreamMats& M, int rc, int& mat) {
    mat = 0;
    int r = rc;
    if (M.n > 1 && r >= M.m[0]) { r -= M.m[0]; mat = 1; if (M.n > 2 && r >= M.m[1]) { r -= M.m[1]; mat = 2; } }
    return r;
}

// where item j of a phase comes from: quants and scales of its two rows (two = false: one row, or two rows of one matrix next to each other as one run)
struct MrItem { const uint8_t* q[2]; const uint16_t* d[2]; unsigned qbytes, dbytes, dspan; bool two; };       // dspan: both rows' scales as one copy, what lies between them included (0: a copy each)
// Where the second row's scales lie behind the first's: beside them, or, where Q8_0 rows are longer than a segment and both fit, as far as in the plane: one copy of
// both and of what lies between them, an item in three copies (11008 x 4096: 14.3 -> 14.0 us, a token 1806 -> 1777; Q4_0 waits for its consumers, larger slots only cost it 0.7 %).
// Slots with room for rows of 14336 too (1152 B) give nothing: four layers of 4096 x 14336 340 -> 342 us, of 5120 x 13824 394 -> 395, 24 of 8192 x 28672 4012 -> 3983
#define MR_SCALES 1024
__device__ __forceinline__ unsigned mr_scale_off(const MrGeo& g, unsigned BB, unsigned dbytes) {
    const unsigned row = 2u * CC_D_STRIDE(g.nb);
    return BB == 32u && g.NSEG > 1 && row + 2u * MK_SEG * 32u <= MR_SCALES ? row : dbytes;
}
__device__ __forceinline__ MrItem mr_item(const StreamMats& M, const MrGeo& g, unsigned BB, int j) {
    MrItem it;
    const int P = j / g.NSEG, sg = j - P * g.NSEG;
    const int u = mr_unit(g, P);
    it.two = u + 1 < g.n_rows;
    int mat = P & 1, matB = mat, rA = g.first + u, rB = rA + (it.two ? 1 : 0);
    if (!g.pair) { const int rc = rA; rA = mr_locate(M, rc, mat); rB = mr_locate(M, rc + (it.two ? 1 : 0), matB); }
    const size_t at = (size_t)sg * (MK_SEG * 32), d_row = (size_t)CC_D_STRIDE(g.nb);
    const unsigned nbe = (unsigned)min(MK_SEG * 32, g.nb - MK_SEG * 32 * sg);
    it.qbytes = nbe * BB;
    it.dbytes = (nbe * 2u + 15u) & ~15u;               // the scale rows are padded to 16 bytes (CC_D_STRIDE): a short last segment copies its padding
    it.q[0] = M.qs[mat] + ((size_t)rA * g.nb + at) * BB; it.d[0] = M.d[mat] + (size_t)rA * d_row + at;
    it.q[1] = M.qs[matB] + ((size_t)rB * g.nb + at) * BB; it.d[1] = M.d[matB] + (size_t)rB * d_row + at;
    if (it.two && g.NSEG == 1 && it.q[1] == it.q[0] + it.qbytes && (const uint8_t*)it.d[1] == (const uint8_t*)it.d[0] + it.dbytes) { it.qbytes *= 2; it.dbytes *= 2; it.two = false; }
    it.dspan = it.two && (const uint8_t*)it.d[1] == (const uint8_t*)it.d[0] + mr_scale_off(g, BB, it.dbytes) ? mr_scale_off(g, BB, it.dbytes) + it.dbytes : 0u;
    return it;
}

// ---- producer warps: run ahead of everybody ---------------------------------------------------------------------------------------------
// All lanes issue (a single issuing thread manages ~1 copy pair per 570 cycles, and the lanes of a warp that have something to issue do it one after another): the thread
// t = 3 * lane + warp owns the items whose number over the whole launch is t mod 96, so that neighbouring items, whose slots come free together, are with different
// warps (32 of them with one: one warp of the three issued at a time; a token of 24 layers of 8192 x 28672 4455 -> 4208 us in Q8_0, 3522 -> 3110 in Q4_0).  It
// decomposes the item into rows and a segment, waits until the slot's previous tenant has been consumed, arms the slot's "full" barrier with the byte
// count, issues the bulk copies (two rows of one matrix that lie next to each other: one for the quants, one for the scales) and publishes the item number in
// the slot's sequence word.  Consumers check that word before they look at the barrier: an mbarrier parity alone cannot tell "this use has not landed" from
// "the use before has not been consumed" when one warp is laps ahead of another.
__device__ void mr_producer(const MkPhase* __restrict__ phases, int n_phases, const MrRing R, unsigned full0, unsigned done0, unsigned ring0,
                            MkPhase* s_pd, volatile unsigned* s_seq, volatile int* s_abort, volatile int* s_dead, volatile int* s_issued, int* s_prod_done, const bool kvpf, const uint8_t* __restrict__ dyn) {
    const int lane = threadIdx.x & 31;
    const int pt = (int)threadIdx.x - MK_THREADS;          // producer thread 0 .. 32 * MR_PRODUCER_WARPS - 1
    for (int i = lane; i < MR_DESC_WORDS; i += 32) ((int*)&s_pd[0])[i] = ((const int*)phases)[i];
    __syncwarp();
    unsigned ent = 0;
    bool dead = false;
    long long t_last = clock64();          // the prefetcher's
    unsigned idle = 0;
    for (int p = 0; p < n_phases && !dead; p++) {
        int nw[MR_DESC_PER_LANE];
#pragma unroll
        for (int j = 0; j < MR_DESC_PER_LANE; j++) { const int i = lane + 32 * j; nw[j] = (p + 1 < n_phases && i < MR_DESC_WORDS) ? ((const int*)(phases + p + 1))[i] : 0; }
        const MkPhase& ph = s_pd[p & 1];
        if (kvpf && ph.type == MK_ATTN) {
            // The attention phase streams a head's K and V rows through 48 KB of shared memory: latency x bytes in flight = 32 GB/s per head
            // (profiles/r02y: +0.04 us per cached position and layer).  The producers reach this table entry while the compute warps are still in
            // the qkv phase: they ask L2 for the cached rows [0, kv_len) of every kv head now, so that the phase's bulk copies hit L2.
            // (rows written by earlier launches: stable; the current token's row never goes through the cache on its way to the phase)
            const AttnArgs& a = ph.at;
            const long long kv_len = ((const long long*)(dyn + ph.dyn_off))[1];
            const unsigned ELT = a.kv_f16 ? 2u : 4u, PIECE = 4096u;
            const size_t head_bytes = (size_t)kv_len * (size_t)a.hd * ELT;
            const long long per_head = (long long)((head_bytes + PIECE - 1) / PIECE), per_cache = per_head * a.n_kv;
            for (long long r = (long long)blockIdx.x * (32 * MR_PRODUCER_WARPS) + pt; r < 2 * per_cache; r += (long long)gridDim.x * (32 * MR_PRODUCER_WARPS)) {
                const long long rr = r >= per_cache ? r - per_cache : r, gk = rr / per_head, piece = rr - gk * per_head;
                const uint8_t* base = (const uint8_t*)(r >= per_cache ? a.vcache : a.kcache) + (size_t)gk * (size_t)a.seq_stride * ELT + (size_t)piece * PIECE;
                const size_t left = head_bytes - (size_t)piece * PIECE;
                const unsigned bytes = (unsigned)(left < PIECE ? left : PIECE) & ~15u;
                if (bytes) asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(base), "r"(bytes) : "memory");
            }
        }
        if (ph.type == MK_MATVEC && ph.act_type != CC_Q8_K) {
            const StreamArgs& A = ph.mv;
            const StreamMats& M = A.mats;
            const MrGeo g = mr_geo(A);
            const unsigned BB = ph.wtype == CC_Q8_0 ? 32u : 16u;
            const unsigned doff = 2u * MK_SEG * 32u * BB;
            const int N = g.groups * g.NSEG;
            if (pt >= MR_ISSUERS) {                // the L2 prefetcher
                const int item = (int)(2u * MK_SEG * 32u * (BB + 2u)), pace = item / MR_L2_RATE, lead = R.nslots + MR_L2_LEAD / item;
                for (int j = 0; j < N && !dead;) {
                    const int issued = __shfl_sync(0xffffffffu, *s_issued, 0) - (int)ent;
                    if (j < issued) { j = min(issued, N); continue; }
                    const long long now = __shfl_sync(0xffffffffu, clock64(), 0);
                    if (t_last < now - 2 * pace) t_last = now - 2 * pace;
                    const int n = min(min(N - j, issued + lead - j), (int)((now - t_last) / pace));          // (two items at most)
                    if (n <= 0) { dead = (++idle & 0x3FFu) == 0 && __any_sync(0xffffffffu, *s_abort || *s_dead); continue; }
                    if (lane < 4 * n) {                // four lanes an item
                        const MrItem im = mr_item(M, g, BB, j + (lane >> 2));
                        const int row = lane & 1;
                        const void* src = lane & 2 ? (row ? (const void*)im.d[1] : (const void*)im.d[0]) : (row ? (const void*)im.q[1] : (const void*)im.q[0]);
                        if (!row || im.two) asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(lane & 2 ? im.dbytes : im.qbytes) : "memory");
                    }
                    __syncwarp();
                    j += n; t_last += (long long)n * pace;
                }
                ent += (unsigned)N;
            } else {
            // a flat loop, one probe of the thread's own slot per trip (a load of the slot's "done" word: no suspension), so a slot is refilled as soon as it is
            // released, not when the slowest lane of a batch is ready
            const int mine = lane * (MR_ISSUERS / 32) + (pt >> 5);
            int j = (mine + MR_ISSUERS - (int)(ent % MR_ISSUERS)) % MR_ISSUERS;
            bool have = false, mydead = false;
            MrItem im = {};
            unsigned e = 0, slot = 0, use = 0, it = 0;
            while (j < N) {
                if (!have) {
                    im = mr_item(M, g, BB, j);
                    e = ent + (unsigned)j; slot = e % (unsigned)R.nslots; use = e / (unsigned)R.nslots;
                    have = true;
                }
                if (!use || (mr_ld_acquire_shared(done0 + 8u * slot) == e - (unsigned)R.nslots + 1u && mr_ld_acquire_shared(done0 + 8u * slot + 4u) == e - (unsigned)R.nslots + 1u)) {      // the slot's previous tenant has been consumed
                    const unsigned fb = full0 + 8u * slot, dst = ring0 + slot * (unsigned)R.slot_bytes;
                    mr_expect_tx(fb, im.dspan ? 2u * im.qbytes + im.dspan : (im.qbytes + im.dbytes) << (im.two ? 1 : 0));
                    mr_bulk_g2s(dst, im.q[0], im.qbytes, fb);
                    if (im.two) mr_bulk_g2s(dst + im.qbytes, im.q[1], im.qbytes, fb);
                    mr_bulk_g2s(dst + doff, im.d[0], im.dspan ? im.dspan : im.dbytes, fb);
                    if (im.two && !im.dspan) mr_bulk_g2s(dst + doff + mr_scale_off(g, BB, im.dbytes), im.d[1], im.dbytes, fb);
                    __threadfence_block();
                    s_seq[slot] = e + 1u;
                    j += MR_ISSUERS; have = false; atomicAdd((int*)s_issued, 1);
                } else if ((++it & 0x3FFu) == 0 && (*s_abort || *s_dead)) { mydead = true; break; }
            }
            dead = __any_sync(0xffffffffu, mydead);
            ent += (unsigned)N;
            }
        }
        __syncwarp();
#pragma unroll
        for (int j = 0; j < MR_DESC_PER_LANE; j++) { const int i = lane + 32 * j; if (i < MR_DESC_WORDS) ((int*)&s_pd[(p + 1) & 1])[i] = nw[j]; }
        __syncwarp();
    }
    if (lane == 0) { __threadfence_block(); atomicAdd(s_prod_done, 1); }
}

// ---- consumer side of a streaming MATVEC phase ------------------------------------------------------------------------------------------
struct MrCons { unsigned full0, done0; const uint8_t* ring; int slot_bytes, nslots; unsigned ent_base; volatile unsigned* s_seq; volatile int* s_dead; unsigned* err_dev; unsigned* err_host; };

// Bounded wait for a slot to fill.  A wait that does not end within 2 s (it takes microseconds) raises the error words (code 4, reported by
// cc_check_async_error) and marks the ring dead for the whole CTA: every later wait returns at once, the launch drains with garbage
// results instead of hanging the GPU.
__device__ __forceinline__ void mr_wait_full(const MrCons& RC, unsigned slot, unsigned e, unsigned parity) {
    const unsigned bar = RC.full0 + 8u * slot;
    volatile unsigned* seq = RC.s_seq + slot;
    if (*seq == e + 1u && mr_try_wait(bar, parity)) return;
    unsigned it = 0;
    unsigned long long t0 = 0;
    for (;;) {
        if (*seq == e + 1u && mr_try_wait(bar, parity)) return;     // entry e has been issued into the slot, and it has landed
        if ((++it & 0xFFFu) != 0) continue;
        if (*RC.s_dead) return;
        const unsigned long long t = cc_globaltimer_ns();
        if (!t0) { t0 = t; continue; }
        if (t - t0 < 2000000000ull) continue;
        *RC.s_dead = 1;
        if (RC.err_dev) atomicExch(RC.err_dev, 4u);
        if (RC.err_host) { *(volatile unsigned*)RC.err_host = 4u; __threadfence_system(); }
        return;
    }
}

// Activation quants in shared memory, per group of 32 blocks: the 16-byte first halves of all 32 blocks, then the second halves (the layout of
// the Q8_0 weight plane) -- lane l reads block 32 g + l with two conflict-free LDS.128 (block-major, 32 bytes apart, is a 2-way bank conflict:
// 64 instead of 32 shared-memory wavefronts per segment, and the ring's throughput is bounded by shared-memory bandwidth)
__device__ __forceinline__ int mr_act_word(int i) {           // i = 4-byte word index in block-major order (block i >> 3, word i & 7)
    const int b = i >> 3, w = i & 7;
    return (b >> 5) * 256 + (w >> 2) * 128 + (b & 31) * 4 + (w & 3);
}
__device__ __forceinline__ int mr_act_int4(int i) {           // i = 16-byte index in block-major order (block i >> 1, half i & 1)
    const int b = i >> 1;
    return (b >> 5) * 64 + (i & 1) * 32 + (b & 31);
}

// The activation of one segment in a lane's registers: its blocks of the four groups.  A warp keeps it for all rows of a phase, so an item costs the shared
// memory 72 wavefronts to read and 68 to fill, and no more: the ring is consumed at shared-memory speed.
template <int TYPE>
struct MrAct { int4 lo[MK_SEG], hi[MK_SEG]; float d[MK_SEG]; int s[TYPE == CC_Q4_0 ? MK_SEG : 1]; };
template <int TYPE>
__device__ __forceinline__ void mr_act_load(MrAct<TYPE>& a, int seg, const int4* aq_l, const float* ad_l, const int* as_l) {
#pragma unroll
    for (int g = 0; g < MK_SEG; g++) {
        const int gi = seg * MK_SEG + g;
        a.lo[g] = aq_l[gi * 64]; a.hi[g] = aq_l[gi * 64 + 32]; a.d[g] = ad_l[gi * 32];
        if constexpr (TYPE == CC_Q4_0) a.s[g] = as_l[gi * 32];
    }
}
// One segment of one row.  `left` = blocks of the row from this segment on: a lane behind them reads what the slot happens to hold (always inside the slot)
// against zero quants and a scale it sets to zero.  The arithmetic is mk_seg_dot's, term by term (bit-identical to matvec_stream.cu).
template <int TYPE>
__device__ __forceinline__ float mr_dot(const uint8_t* q, const uint16_t* d, int left, int last_half_off, int lane, const MrAct<TYPE>& act) {
    constexpr int GB = TYPE == CC_Q8_0 ? 1024 : 512;
    float acc = 0.0f;
#pragma unroll
    for (int g = 0; g < MK_SEG; g++) {
        const int4 w = *(const int4*)(q + lane * 16 + g * GB);
        const uint16_t s = g * 32 + lane < left ? d[g * 32 + lane] : (uint16_t)0;
        int sum;
        if constexpr (TYPE == CC_Q8_0) {
            const int4 w1 = *(const int4*)(q + lane * 16 + g * GB + (left <= (g + 1) * 32 ? last_half_off : 512));
            sum = mk_dp16(w, act.lo[g]) + mk_dp16(w1, act.hi[g]);
        } else {
            const int4 lo = make_int4(w.x & 0x0F0F0F0F, w.y & 0x0F0F0F0F, w.z & 0x0F0F0F0F, w.w & 0x0F0F0F0F);
            const int4 hi = make_int4((w.x >> 4) & 0x0F0F0F0F, (w.y >> 4) & 0x0F0F0F0F, (w.z >> 4) & 0x0F0F0F0F, (w.w >> 4) & 0x0F0F0F0F);
            sum = mk_dp16(lo, act.lo[g]) + mk_dp16(hi, act.hi[g]) - 8 * act.s[g];
        }
        acc += (float)sum * h2f_bits(s) * act.d[g];
    }
    return acc;
}

// Fused prologue: [exchange reduction] + [rms_norm * w] + Q8_0 quantisation of x by EVERY CTA: thread t owns the float4 chunks t, t + 512, ... (the
// canonical reduction order of common.cuh, and 8 consecutive threads = one 32-block).  All chunks of a thread are asked for at once, into shared memory, and the
// loops over them are short: the phases of a layer do not stay in the near instruction caches, and the kernel's 96 registers have no room for a row (a spilled
// register is a trip to L2 here, the ring leaves no L1).  The divisions are multiplications with the same bits (quotients.cuh).
#define MR_ROW_PIECE 12288             // elements (whole passes of 512 threads x 4)
template <int TYPE>
__device__ __forceinline__ void mr_prologue(const MkPhase& ph, int k, int nbp, int* s_q32, float* s_d, int* s_s, float* s_red, float4* s_x, const CommDev& comm, unsigned xseq) {
    const int n4 = k >> 2, nch = nbp << 3;                              // chunks of the row; with the zeros behind it (nbp % 128 == 0: whole passes of 512 threads)
    const int piece = min(n4, MR_ROW_PIECE / 4);                        // a longer row goes through the staging area in pieces
    const float* nw = ph.norm_w;
    float4* s_w = s_x + piece;
    const float* xbase = ph.red_n ? comm.data[comm.rank] + (size_t)(xseq & 1u) * CC_COMM_MAX_RANKS * CC_COMM_MAX_ELEMS : ph.x;
    auto fetch = [&](int i0) {
        const int n = min(piece, n4 - i0);
#pragma unroll 2
        for (int i = threadIdx.x; i < n; i += MK_THREADS) {
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(s_x + i)), "l"((const float4*)xbase + i0 + i) : "memory");
            if (nw) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(s_w + i)), "l"((const float4*)nw + i0 + i) : "memory");
        }
        asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");     // (a thread reads only what it asked for itself)
        if (ph.red_n) {                                                 // sum over ranks in rank order (+ residual): comm.cu
#pragma unroll 1
            for (int i = threadIdx.x; i < n; i += MK_THREADS) {
                float4 a = s_x[i];
                for (int p = 1; p < comm.world; p++) {
                    const float4 t = __ldcg((const float4*)(xbase + (size_t)p * CC_COMM_MAX_ELEMS) + i0 + i);
                    a.x += t.x; a.y += t.y; a.z += t.z; a.w += t.w;
                }
                if (ph.red_res) { const float4 r = __ldcg((const float4*)ph.red_res + i0 + i); a.x += r.x; a.y += r.y; a.z += r.z; a.w += r.w; }
                s_x[i] = a;
            }
        }
    };
    float rms = 1.0f, rr = 1.0f;
    if (nw) {
        float ss = 0.0f;
        for (int i0 = 0; i0 < n4; i0 += piece) {
            fetch(i0);
#pragma unroll 2
            for (int i = threadIdx.x; i < min(piece, n4 - i0); i += MK_THREADS) ss += cc_sq4(s_x[i]);
        }
        ss = warp_sum(ss);
        if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = ss;
        MK_SYNC();
        float t = 0.0f;
#pragma unroll
        for (int w = 0; w < MK_WARPS; w++) t += s_red[w];
        rms = sqrtf(t / (float)k + ph.eps);
        rr = 1.0f / rms;
    }
    const bool rms_ok = cc_quot_range(rms);
    int i0 = 0;
    if (!nw || n4 > piece) fetch(0);
    // chunk i = 4 elements of block i >> 3.  512 chunks on are 64 blocks on: two groups of 32 in s_q32
    int* out = s_q32 + mr_act_word(threadIdx.x);
#pragma unroll 1
    for (int i = threadIdx.x; i < nch; i += MK_THREADS, out += 512) {
        if (i - i0 >= piece && i0 + piece < n4) { i0 += piece; fetch(i0); }             // (whole passes of 512 threads: all of them together)
        const bool live = i < n4;
        if (!__any_sync(0xffffffffu, live)) {                           // behind the row: zeros (a segment is 128 blocks, a row of 288 has nine)
            *out = 0;
            if ((threadIdx.x & 7) == 0) { s_d[i >> 3] = 0.0f; if constexpr (TYPE == CC_Q4_0) s_s[i >> 3] = 0; }
            continue;
        }
        float4 v = live ? s_x[i - i0] : make_float4(0, 0, 0, 0);
        if (ph.orig && blockIdx.x == 0 && live) ((float4*)ph.orig)[i] = v;              // Tensor::dup of the un-normalised row (llama2.rs:227,607)
        const float4 x = v;
        bool sure = true;
        if (nw && live) {
            const float4 w = s_w[i - i0];
            sure = rms_ok && cc_quot_no_tiny(v.x, v.y, v.z, v.w);
            v = make_float4(cc_quot_by(v.x, rms, rr) * w.x, cc_quot_by(v.y, rms, rr) * w.y, cc_quot_by(v.z, rms, rr) * w.z, cc_quot_by(v.w, rms, rr) * w.w);
        }
        float amax = fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w)));
        const float nan = (v.x + v.y) + (v.z + v.w);                    // (the maximum leaves one out; infinities are out of range)
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
        if (!live) amax = 1.0f;
        sure = sure && cc_quot_range(amax) && nan == nan;
        float d = cc_q8_0_scale(amax), rcp;
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rcp) : "f"(d));        // within one unit in the last place
        const float half = 0.5f * d;
        int q0 = cc_q8_0_quant(v.x, d, half, rcp), q1 = cc_q8_0_quant(v.y, d, half, rcp), q2 = cc_q8_0_quant(v.z, d, half, rcp), q3 = cc_q8_0_quant(v.w, d, half, rcp);
        if (__any_sync(0xffffffffu, !sure)) {                           // rare: the whole warp's chunk with its divisions
            v = x;
            if (nw && live) { const float4 w = s_w[i - i0]; v = make_float4((v.x / rms) * w.x, (v.y / rms) * w.y, (v.z / rms) * w.z, (v.w / rms) * w.w); }
            amax = fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w)));
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
            d = amax / 127.0f;
            q0 = live ? __float2int_rz(v.x / d) : 0; q1 = live ? __float2int_rz(v.y / d) : 0; q2 = live ? __float2int_rz(v.z / d) : 0; q3 = live ? __float2int_rz(v.w / d) : 0;
        }
        *out = (int)__byte_perm(__byte_perm((unsigned)q0, (unsigned)q1, 0x0040), __byte_perm((unsigned)q2, (unsigned)q3, 0x0040), 0x5410);
        if constexpr (TYPE == CC_Q4_0) {
            int sq = q0 + q1 + q2 + q3;
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
            if ((threadIdx.x & 7) == 0) s_s[i >> 3] = sq;
        }
        if ((threadIdx.x & 7) == 0) s_d[i >> 3] = live ? __half2float(__float2half_rn(d)) : 0.0f;
    }
}

// Lanes' sums are added up behind the row loop, all rows of the CTA at once, where they find room in shared memory (ph.ring_parts, decided by the host for all CTAs
// alike).  One segment: a thread adds up a row's 32 (the butterfly took 320 of 1350 cycles a row).  Several: warps keep to one segment, so that its activation stays in
// registers, and a warp adds up a row's.  Else a warp takes a row's segments one after another, reads the activation for each and adds up itself.
// The room is taken from the ring.  30 KB are 232 rows of one segment (a vocabulary of 32000; one of 128256 comes at 7.3 TB/s all the same).  Rows of five segments and more
// have 56 KB (8192 rows of eight): without it the ring holds the items of two or three pairs of rows, and as many pairs of warps work: 8192 x 28672 58.6 -> 45.2 us in
// Q8_0, 42.7 -> 34.4 in Q4_0; four layers of 6144 x 20480 494 -> 476 and 423 -> 431 (five segments, eight pairs of warps).  86 KB (12288 x 32768) cost a
// token of two such layers more than it gave, 680 -> 742.
#define MR_PART_BYTES(nseg) ((nseg) > 4 ? 57344 : 30720)
// shared memory of the phase: quants [nbp * 32] | f32 scales [nbp] | block sums [nbp] | reduction scratch 256 B | sums of the CTA's virtual rows | lanes' sums | fused prologue (over the sums): the row and its norm weights
template <int TYPE>
__device__ void phase_matvec_ring(const MkPhase& ph, uint8_t* smem, const uint16_t* exp_lut, MrCons& RC, const CommDev& comm, unsigned xseq, unsigned long long* stamp1) {
    const StreamArgs& A = ph.mv;
    const int k = A.k;
    const MrGeo g = mr_geo(A);
    const int nb = g.nb, NSEG = g.NSEG;
    const bool pair = g.pair;
    const int nbp = NSEG * MK_SEG * 32;
    int8_t* s_q = (int8_t*)smem;
    float* s_d = (float*)(smem + (size_t)nbp * 32);
    int* s_s = (int*)(smem + (size_t)nbp * 32 + (size_t)nbp * 4);
    float* s_red = (float*)(smem + (size_t)nbp * 40);
    float* s_sum = (float*)(smem + (size_t)nbp * 40 + 256);
    const int vrows = pair ? 2 * g.n_rows : g.n_rows;
    float* s_part = s_sum + ph.ring_sums;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const StreamMats& M = A.mats;
    if (ph.x) {
        mr_prologue<TYPE>(ph, k, nbp, (int*)s_q, s_d, s_s, s_red, (float4*)s_sum, comm, xseq);
    } else {   // stage the quantised activation (written by other CTAs in the previous phase: L2 loads)
        const uint8_t* act = (const uint8_t*)A.act;
        const int4* gq = (const int4*)act;
        int4* sq4 = (int4*)s_q;
        const float* gd = (const float*)(act + ((k + 15) & ~15));
        const int* gs = (const int*)(act + ((k + 15) & ~15) + ((nb * 4 + 15) & ~15));
        if (nbp <= MK_THREADS) {           // every load of the thread is issued before its first store (one L2 round trip, not three)
            const int i0 = threadIdx.x, i1 = threadIdx.x + MK_THREADS;
            const int4 z4 = make_int4(0, 0, 0, 0);
            const int4 qa = i0 < nb * 2 ? __ldcg(gq + i0) : z4, qb = i1 < nb * 2 ? __ldcg(gq + i1) : z4;
            const float dv = i0 < nb ? __ldcg(gd + i0) : 0.0f;
            int sv = 0;
            if constexpr (TYPE == CC_Q4_0) sv = i0 < nb ? __ldcg(gs + i0) : 0;
            if (i0 < nbp * 2) sq4[mr_act_int4(i0)] = qa;
            if (i1 < nbp * 2) sq4[mr_act_int4(i1)] = qb;
            if (i0 < nbp) { s_d[i0] = dv; if constexpr (TYPE == CC_Q4_0) s_s[i0] = sv; }
        } else {
            for (int i = threadIdx.x; i < nbp * 2; i += MK_THREADS) sq4[mr_act_int4(i)] = i < nb * 2 ? __ldcg(gq + i) : make_int4(0, 0, 0, 0);
            for (int i = threadIdx.x; i < nbp; i += MK_THREADS) {
                s_d[i] = i < nb ? __ldcg(gd + i) : 0.0f;
                if constexpr (TYPE == CC_Q4_0) s_s[i] = i < nb ? __ldcg(gs + i) : 0;
            }
        }
    }
    MK_SYNC();
    if (stamp1) *stamp1 = globaltimer_ns();
    const int4* aq_l = (const int4*)s_q + lane;
    const float* ad_l = s_d + lane;
    const int* as_l = s_s + lane;
    // Warps 2 i and 2 i + 1 take the two rows of an item.  One warp on both rows held sixteen of the twenty slots at a time, so few copies were under way
    const int duo = warp >> 1, half = warp & 1;
    const bool parts = ph.ring_parts != 0, split = parts && NSEG > 1;
    const int s0 = split ? duo % NSEG : 0, ns = split ? 1 : NSEG;
    const int P0 = split ? duo / NSEG : duo, dP = split ? (MK_WARPS / 2 - s0 + NSEG - 1) / NSEG : MK_WARPS / 2;
    constexpr unsigned DOFF = 2u * MK_SEG * (TYPE == CC_Q8_0 ? 1024u : 512u);
    const unsigned NS = (unsigned)RC.nslots;
    MrAct<TYPE> act;
    mr_act_load<TYPE>(act, s0, aq_l, ad_l, as_l);
    unsigned e = RC.ent_base + (unsigned)(P0 * NSEG + s0), slot = e % NS, par = (e / NS) & 1u;
    for (int P = P0; P < g.groups; P += dP) {
        const int u = mr_unit(g, P) + half, v = pair ? 2 * u + (P & 1) : u;
        const bool row = u < g.n_rows;
        float acc = 0.0f;
        for (int s = 0; s < ns; s++) {
            const int sg = s0 + s;
            if (ns > 1) mr_act_load<TYPE>(act, sg, aq_l, ad_l, as_l);
            const int left = nb - sg * (MK_SEG * 32), nbe = min(MK_SEG * 32, left);
            mr_wait_full(RC, slot, e, par);
            float part = 0.0f;
            if (row) {
                const uint8_t* sp = RC.ring + (size_t)slot * RC.slot_bytes;
                part = mr_dot<TYPE>(sp + (half ? (unsigned)nbe * (TYPE == CC_Q8_0 ? 32u : 16u) : 0u), (const uint16_t*)(sp + DOFF + (half ? mr_scale_off(g, TYPE == CC_Q8_0 ? 32u : 16u, (unsigned)((nbe * 2 + 15) & ~15)) : 0u)), left,
                                    g.last_half_off, lane, act);
            }
            acc += part;
            __syncwarp();
            if (lane == 0) mr_release(RC.done0 + 8u * slot + 4u * (unsigned)half, e + 1u, part);
            const unsigned step = s + 1 < ns ? 1u : (unsigned)((dP - 1) * NSEG) + (split ? (unsigned)NSEG : 1u);
            e += step; slot += step;
            while (slot >= NS) { slot -= NS; par ^= 1u; }
        }
        if (!row) continue;
        if (split) s_part[(v * NSEG + s0) * 32 + lane] = acc;
        else if (parts) s_part[v * 33 + lane] = acc;
        else { const float r = warp_sum(acc); if (lane == 0) s_sum[v] = r; }
    }
    RC.ent_base += (unsigned)(g.groups * NSEG);
    float res = 0.0f;                                                  // + residual (llama2.rs:266,636)
    if (A.epilogue == 1 && (int)threadIdx.x < g.n_rows) res = ldcg_f(A.residual + g.first + threadIdx.x);
    MK_SYNC();
    if (split) {                                                       // a row's segments in their order, then the butterfly
        for (int v = warp; v < vrows; v += MK_WARPS) {
            float acc = 0.0f;
            for (int s = 0; s < NSEG; s++) acc += s_part[((size_t)v * NSEG + s) * 32 + lane];
            const float r = warp_sum(acc);
            if (lane == 0) s_sum[v] = r;
        }
        MK_SYNC();
    }
    // a row per thread, neighbouring rows side by side in memory; gate and up of a unit on neighbouring threads
    for (int v = threadIdx.x; v - lane < vrows; v += MK_THREADS) {
        float r = 0.0f;
        if (v < vrows) {
            if (parts && !split) {                                     // the butterfly's sum, its pairs in its order (stride 33: no bank conflicts)
                const float* p = s_part + v * 33;
                float t[16];
#pragma unroll
                for (int i = 0; i < 16; i++) t[i] = p[i] + p[i + 16];
#pragma unroll
                for (int o = 8; o > 0; o >>= 1)
#pragma unroll
                    for (int i = 0; i < o; i++) t[i] += t[i + o];
                r = t[0];
            } else r = s_sum[v];
        }
        const float up = __shfl_down_sync(0xffffffffu, r, 1);
        if (v >= vrows) continue;
        if (pair) {                                                    // silu(gate) * up
            if (!(v & 1)) M.out[0][g.first + (v >> 1)] = (r / (1.0f + h2f_bits(exp_lut[f2h_bits(-r)]))) * up;
        } else if (A.epilogue == 1) {
            if (v >= MK_THREADS) res = ldcg_f(A.residual + g.first + v);
            M.out[0][g.first + v] = r + res;
        } else if (A.epilogue == 3) s_sum[v] = r;
        else {
            int mat;
            const int rr = mr_locate(M, g.first + v, mat);
            float* o = mat == 0 ? M.out[0] : mat == 1 ? M.out[1] : M.out[2];
            o[rr] = r;
        }
    }
    if (A.epilogue == 3) {
        // the CTA's block of partial rows -> slot[rank] of every GPU's exchange window: warp p serves peer p with coalesced 16-byte
        // NVLink stores (mega.cu)
        MK_SYNC();
        if (warp < comm.world) {
            const size_t off = ((size_t)((xseq + 1u) & 1u) * CC_COMM_MAX_RANKS + comm.rank) * CC_COMM_MAX_ELEMS + g.first;
            for (int c4 = lane * 4; c4 < g.n_rows; c4 += 128) *(float4*)(comm.data[warp] + off + c4) = *(const float4*)(s_sum + c4);
        }
    }
}

template <bool GEN>
__global__ void __launch_bounds__(MR_THREADS, 1) mega_ring_kernel(const MkPhase* __restrict__ phases, int n_phases, const uint8_t* dyn, unsigned* bar,
                                                                  const uint16_t* exp_lut, unsigned long long* prof, int flags, int wtop_off, unsigned* err_host,
                                                                  const __grid_constant__ CommDev comm, const __grid_constant__ MrRing R) {
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ float s_red[MK_WARPS];
    __shared__ MkPhase s_phs[2];             // phase descriptors of the compute warps, double-buffered
    __shared__ MkPhase s_pd[MR_PRODUCER_WARPS][2];      // every producer warp keeps its own copies (it runs phases ahead, at its own pace)
    __shared__ int s_abort;
    __shared__ int s_prod_done;
    __shared__ int s_ring_dead;
    __shared__ int s_issued;                 // items under way or landed since the launch began
    __shared__ __align__(8) unsigned long long s_abar[AT_NBUF];
    __shared__ __align__(8) unsigned long long s_full[MR_MAX_SLOTS];
    __shared__ unsigned s_done[2 * MR_MAX_SLOTS]; // item number + 1 of the slot's last consumed tenant, a word per row
    __shared__ unsigned s_seq[MR_MAX_SLOTS];      // item number + 1 of the slot's current tenant
    unsigned apar = 0u;
    const unsigned abar0 = (unsigned)__cvta_generic_to_shared(&s_abar[0]);
    const unsigned full0 = (unsigned)__cvta_generic_to_shared(&s_full[0]);
    const unsigned done0 = (unsigned)__cvta_generic_to_shared(&s_done[0]);
    if (threadIdx.x == 0) {
        for (int i = 0; i < AT_NBUF; i++) mbar_init(abar0 + 8u * i, 1u);
        for (int i = 0; i < R.nslots; i++) { mbar_init(full0 + 8u * i, 1u); s_done[2 * i] = 0u; s_done[2 * i + 1] = 0u; s_seq[i] = 0u; }
        s_abort = 0; s_prod_done = 0; s_ring_dead = 0; s_issued = 0;
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();                         // the only barrier all 640 threads share
    if (threadIdx.x >= MK_THREADS) {
        mr_producer(phases, n_phases, R, full0, done0, (unsigned)__cvta_generic_to_shared(smem + R.ring_off), s_pd[(threadIdx.x - MK_THREADS) >> 5], s_seq, &s_abort, &s_ring_dead, &s_issued, &s_prod_done,
                    (flags & MK_F_KVPF) != 0, dyn);
        return;
    }
    MrCons RC;
    RC.full0 = full0; RC.done0 = done0; RC.ring = smem + R.ring_off; RC.slot_bytes = R.slot_bytes; RC.nslots = R.nslots; RC.ent_base = 0u;
    RC.s_seq = s_seq; RC.s_dead = &s_ring_dead; RC.err_dev = &bar[MK_BAR_ERR]; RC.err_host = err_host;
    AtPre at_pre = {0, 0, 0.0f, 0.0f};
    uint8_t* work = smem;
    float* s_w = (float*)(smem + wtop_off);  // generic phases: staging of the norm weights
    unsigned gen = 0;
    if (threadIdx.x == MK_BAR_THREAD) gen = ld_acquire_u32(&bar[32]);
    unsigned xseq = comm.world > 0 ? *comm.seq : 0u;
    for (int i = threadIdx.x; i < MR_DESC_WORDS; i += MK_THREADS) ((int*)&s_phs[0])[i] = ((const int*)phases)[i];
    for (int p = 0; p < n_phases; p++) {
        const bool stamp = prof && blockIdx.x == 0 && threadIdx.x == 0;
        if (stamp) { prof[p * MK_PROF_SLOTS] = globaltimer_ns(); prof[p * MK_PROF_SLOTS + 1] = 0; prof[p * MK_PROF_SLOTS + 4] = 0; prof[p * MK_PROF_SLOTS + 5] = 0; }
        MK_SYNC();                           // descriptor p is in shared memory (stored one phase ago)
        const MkPhase& s_ph = s_phs[p & 1];
        if (p == 0 && s_ph.type == MK_ATTN) at_pre = at_ask(s_ph, (float*)work, dyn, abar0, R.at_ch);
        static_assert(sizeof(MkPhase) / 4 <= MK_THREADS, "descriptor does not fit one word per thread");
        int desc_w = 0;
        if (p + 1 < n_phases && threadIdx.x < sizeof(MkPhase) / 4) desc_w = ((const int*)(phases + p + 1))[threadIdx.x];
        unsigned long long* st1 = stamp ? prof + p * MK_PROF_SLOTS + 1 : nullptr;
        switch (s_ph.type) {
        case MK_NORMQ: phase_normq(s_ph, s_red); break;
        case MK_MATVEC:
            if (GEN && s_ph.act_type == CC_Q8_K) {
                switch (s_ph.wtype) {
                case CC_Q2_K: phase_matvec_generic<TQ2_K>(s_ph, work, s_w, false, false, exp_lut, MK_GENERIC_PIPE_ARG st1); break;
                case CC_Q3_K: phase_matvec_generic<TQ3_K>(s_ph, work, s_w, false, false, exp_lut, MK_GENERIC_PIPE_ARG st1); break;
                case CC_Q4_K: phase_matvec_generic<TQ45_K<false>>(s_ph, work, s_w, false, false, exp_lut, MK_GENERIC_PIPE_ARG st1); break;
                case CC_Q5_K: phase_matvec_generic<TQ45_K<true>>(s_ph, work, s_w, false, false, exp_lut, MK_GENERIC_PIPE_ARG st1); break;
                case CC_Q6_K: phase_matvec_generic<TQ6_K>(s_ph, work, s_w, false, false, exp_lut, MK_GENERIC_PIPE_ARG st1); break;
                default: phase_matvec_generic<TQ8_K>(s_ph, work, s_w, false, false, exp_lut, MK_GENERIC_PIPE_ARG st1); break;
                }
                break;
            }
            if (s_ph.wtype == CC_Q8_0) phase_matvec_ring<CC_Q8_0>(s_ph, work, exp_lut, RC, comm, xseq, st1);
            else phase_matvec_ring<CC_Q4_0>(s_ph, work, exp_lut, RC, comm, xseq, st1);
            break;
        case MK_ATTN:
            if (s_ph.at.kv_f16) phase_attn<true>(s_ph, (float*)work, s_red, at_pre, exp_lut, abar0, apar, R.at_ch);
            else phase_attn<false>(s_ph, (float*)work, s_red, at_pre, exp_lut, abar0, apar, R.at_ch);
            at_pre.jobs = 0;
            break;
        case MK_ROWS: phase_rows(s_ph, dyn); break;
        case MK_REDUCE: phase_reduce(s_ph, comm, xseq, false); break;
        case MK_GATHER: phase_reduce(s_ph, comm, xseq, true); break;
        case MK_ARGMAX: phase_argmax(s_ph, dyn, s_red); break;
        }
        if (stamp) prof[p * MK_PROF_SLOTS + 2] = globaltimer_ns();
        if (p + 1 < n_phases && threadIdx.x < sizeof(MkPhase) / 4) ((int*)&s_phs[(p + 1) & 1])[threadIdx.x] = desc_w;
        const bool more = p + 1 < n_phases;
        const bool xg = s_ph.xgpu != 0;
        if ((flags & MK_F_TESTSTALL) && p == 2 && blockIdx.x == gridDim.x - 1) { if (threadIdx.x == 0) s_abort = 1; break; }     // test hook: this CTA deserts
        if (more) grid_barrier_arrive(bar, gridDim.x, gen, xg, (flags & MK_F_SYSFENCE) != 0);
        if (more) {
            const MkPhase& nx = s_phs[(p + 1) & 1];
            if (nx.type == MK_ATTN) at_pre = at_ask(nx, (float*)work, dyn, abar0, R.at_ch);
            // the norm weights of the next prologue were last read a token ago and come from HBM: a line of them per CTA into
            // L2 now (0.8 % of a 7B token)
            else if (nx.type == MK_MATVEC && nx.norm_w && threadIdx.x < 8)
                for (int i = ((int)blockIdx.x * 8 + (int)threadIdx.x) * 32; i < nx.mv.k; i += (int)gridDim.x * 256) asm volatile("prefetch.global.L2 [%0];" ::"l"(nx.norm_w + i));
        }
        if (stamp) prof[p * MK_PROF_SLOTS + 3] = globaltimer_ns();
        if (more) {
            grid_barrier_wait(bar, gridDim.x, gen, comm, xg ? xseq + 1u : 0u, (flags & MK_F_POLLCNT) != 0, &s_abort, err_host);
            gen++; if (xg) xseq++;
            if (s_abort) break;              // a barrier timed out: bail out, the host reports it
        }
    }
    if (comm.world > 0 && blockIdx.x == 0 && threadIdx.x == 0) *comm.seq = xseq;
    if (prof && blockIdx.x == 0 && threadIdx.x == 0) prof[n_phases * MK_PROF_SLOTS] = globaltimer_ns();
    // a launch that gave up: the producer stops at its next look at s_abort; bulk copies it has already issued must land before
    // the CTA's shared memory goes away
    MK_SYNC();
    if ((s_abort || s_ring_dead) && threadIdx.x == 0) {
        at_drain(at_pre.jobs, abar0, apar);
        while (*(volatile int*)&s_prod_done < MR_PRODUCER_WARPS) {}
        for (unsigned sl = 0; sl < (unsigned)R.nslots; sl++) {               // every slot's latest tenant has landed
            const unsigned q = *(volatile unsigned*)&s_seq[sl];
            if (q) mbar_wait(full0 + 8u * sl, ((q - 1u) / (unsigned)R.nslots) & 1u);
        }
    }
}

// ---- host side ---------------------------------------------------------------------------------------------------------------------------
// a streaming MATVEC phase can be fed by bulk copies when every segment is a whole number of 16-byte units at a 16-byte aligned address
// (always, since the scale rows are padded: CC_D_STRIDE; the check keeps the pointer alignment honest)
bool cc_mega_ring_phase_ok(const MkPhase& ph) {
    if (ph.type != MK_MATVEC || ph.act_type == CC_Q8_K) return true;
    if (ph.wtype != CC_Q8_0 && ph.wtype != CC_Q4_0) return false;
    if (ph.mv.k % 32) return false;
    for (int t = 0; t < ph.mv.mats.n; t++)
        if (((uintptr_t)ph.mv.mats.qs[t] | (uintptr_t)ph.mv.mats.d[t]) & 15u) return false;
    return true;
}
int cc_mega_ring_at_ch(const MkPhase& ph) {       // 48 KB of cache rows in flight per head either way (CRABML_RING_ATCH: developer A/B)
    static const int env = getenv("CRABML_RING_ATCH") ? atoi(getenv("CRABML_RING_ATCH")) : 0;
    if (env >= 8 && env <= 64) return env;
    return ph.at.kv_f16 ? 64 : 32;
}
size_t cc_mega_ring_layout(MkPhase& ph, int ctas) {
    if (ph.type == MK_MATVEC && ph.act_type == CC_Q8_K) return cc_mega_smem_for_phase(ph);
    if (ph.type == MK_MATVEC) {
        const size_t k = (size_t)ph.mv.k, nb = k / 32, GR = (nb + 31) / 32, NSEG = (GR + MK_SEG - 1) / MK_SEG, nbp = NSEG * MK_SEG * 32;
        const size_t m = ph.mv.epilogue == 2 ? (size_t)ph.mv.mats.m[0] : (size_t)ph.mv.mats.m[0] + (ph.mv.mats.n > 1 ? ph.mv.mats.m[1] : 0) + (ph.mv.mats.n > 2 ? ph.mv.mats.m[2] : 0);
        const size_t rows = (m + (size_t)ctas - 1) / (size_t)ctas, most = ph.mv.epilogue == 2 ? 2 * rows : ph.mv.epilogue == 3 ? (rows + 3) & ~(size_t)3 : rows;      // the CTA with the most rows: mr_geo
        const size_t own = ((most + 31) & ~(size_t)31) * 4, parts = NSEG == 1 ? most * 132 : most * NSEG * 128;
        ph.ring_sums = (int)(own / 4); ph.ring_parts = NSEG <= MK_WARPS / 2 && parts <= MR_PART_BYTES(NSEG);
        const size_t sums = own + (ph.ring_parts ? parts : 0);
        const size_t row = ph.x ? (k < MR_ROW_PIECE ? k : MR_ROW_PIECE) * 4 * (ph.norm_w ? 2 : 1) : 0;
        return nbp * 40 + 256 + (sums > row ? sums : row);
    }
    if (ph.type == MK_ATTN) return (size_t)(3 * ph.at.hd + ((ph.at.max_len + 8 + 3) & ~3)) * 4 + (size_t)AT_NBUF * cc_mega_ring_at_ch(ph) * ph.at.hd * (ph.at.kv_f16 ? 2 : 4) + 64;
    return 1024;
}
// slots the ring would get beside a working area of `smem_work` (+ `smem_wstage`) bytes; lazy.cu falls back to the register-pipe kernel
// (mega.cu) below MR_MIN_SLOTS -- e.g. a 32 K-token context, whose attention phase needs 128 KB for the score row alone
#define MR_MIN_SLOTS 6
static size_t mr_ring_off(size_t smem_work, size_t smem_wstage) { return ((((smem_work + 15) & ~(size_t)15) + smem_wstage) + 127) & ~(size_t)127; }
int cc_mega_ring_slots(size_t smem_work, size_t smem_wstage, int slot_bytes, bool generic) {
    cudaFuncAttributes fa;
    if (cudaFuncGetAttributes(&fa, generic ? mega_ring_kernel<true> : mega_ring_kernel<false>) != cudaSuccess) { cudaGetLastError(); return 0; }
    const size_t cap = 227 * 1024 - fa.sharedSizeBytes, off = mr_ring_off(smem_work, smem_wstage);
    if (slot_bytes <= 0 || off >= cap) return 0;
    const size_t n = (cap - off) / (size_t)slot_bytes;
    return (int)(n > MR_MAX_SLOTS ? MR_MAX_SLOTS : n);
}
bool cc_mega_ring_fits(size_t smem_work, size_t smem_wstage, int slot_bytes, bool generic) { return cc_mega_ring_slots(smem_work, smem_wstage, slot_bytes, generic) >= MR_MIN_SLOTS; }

int cc_launch_mega_ring(cc_device* dev, const MkPhase* phases_dev, int n_phases, const uint8_t* dyn_dev, unsigned* bar_dev, size_t smem_work, size_t smem_wstage,
                        unsigned long long* prof, const CommDev* comm, bool generic, int slot_bytes, int at_ch, int flags) {
    auto kern = generic ? mega_ring_kernel<true> : mega_ring_kernel<false>;
    cudaFuncAttributes fa;
    CC_CUDA(dev, cudaFuncGetAttributes(&fa, kern));
    const size_t wtop = (smem_work + 15) & ~(size_t)15;
    const size_t ring_off = (wtop + smem_wstage + 127) & ~(size_t)127;
    const size_t cap = 227 * 1024 - fa.sharedSizeBytes;
    CC_REQUIRE(dev, ring_off + 4 * (size_t)slot_bytes <= cap, "megakernel: the phases leave no room for the weight ring (%zu bytes of working area)", ring_off);
    int nslots = (int)((cap - ring_off) / (size_t)slot_bytes);
    if (nslots > MR_MAX_SLOTS) nslots = MR_MAX_SLOTS;
    if (const char* e = getenv("CRABML_RING_SLOTS")) { const int v = atoi(e); if (v >= 2 && v < nslots) nslots = v; }      // developer A/B
    const size_t smem = ring_off + (size_t)nslots * slot_bytes;
    CC_CUDA(dev, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int max_ctas_per_sm = 0;
    CC_CUDA(dev, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&max_ctas_per_sm, kern, MR_THREADS, smem));
    CC_REQUIRE(dev, max_ctas_per_sm >= 1, "megakernel (ring) does not fit on an SM");
    CommDev cd;
    memset(&cd, 0, sizeof(cd));
    if (comm) cd = *comm;
    MrRing R;
    R.ring_off = (int)ring_off; R.slot_bytes = slot_bytes; R.nslots = nslots; R.at_ch = at_ch;
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3((unsigned)dev->sm_count); cfg.blockDim = dim3(MR_THREADS); cfg.dynamicSmemBytes = smem; cfg.stream = dev->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = getenv("CRABML_MEGA_COOP") ? 1 : 0;          // see cc_launch_mega
    cfg.attrs = attr; cfg.numAttrs = 1;
    const uint16_t* lut = dev->exp_lut;
    CC_CUDA(dev, cudaLaunchKernelEx(&cfg, kern, phases_dev, n_phases, dyn_dev, bar_dev, lut, prof, flags, (int)wtop, dev->err_host, (const CommDev)cd, (const MrRing)R));
    CC_LAUNCH_CHECK(dev);
    return CC_OK;
}
