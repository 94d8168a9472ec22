// flat_round.cuh -- one collision round of the warp-flattened mesh step, shared
// by the single-job step kernel (flat.cu) and the multi-job batch kernel
// (batch.cu).
//
// Semantics: rfdougherty/dSim dSim3/src/spinKernelCpu.cpp:198-337 (the
// collision search over the cells of the sub-segment's box, nearest hit of the
// first reference cell with a hit, last-hit triangle excluded).  The lanes'
// fine-cell boxes form one flat list of cells (a prefix sum; an element's owner
// from a mask of starts and a rank table, flat_starts); 32 cells at a time are
// looked up and those whose slab the sub-segment may meet are kept.  The kept
// cells' records form flat lists in blocks of 32 cells, tested 64 records at a
// time against their owners' sub-segments (segment table in shared memory);
// records past the plane test are queued and finished 32 at a time.  Hits are
// filed in the owner's shared-memory slots.  An owner with one hit of a triangle
// that every reference cell it enters lists takes it; others choose by the
// reference's walk over its cells (exact reference-grid scan when the slots
// overflowed).
//
// Bound by instruction issue and L2 latency together (400,000 spins on 640,000
// triangles, 5 blocks per SM: issue 47 %, long-scoreboard stalls 4.0 of 9.0 cycles
// an instruction, DRAM idle), so by how many warps an SM can hold.  Warp
// instructions per step of 32 spins went 3031 -> 2513 (slabs) -> 2164 (owners by
// mask and rank instead of five-shuffle searches, no integer division, full
// windows, one copy of the exact test, no walk over cells for nine hits in ten):
// 6.6e9 -> 9.1e9 spin-steps/s there, 6.8e9 -> 9.4e9 for 1M spins on 2.56M
// triangles; then 11.1e9 and 10.8e9 with a lane's state in shared memory
// (LaneState), 7 blocks per SM and the spins dealt out (kDealWarps).  All on tubes
// that do not overlap.  Where they do, single spins caught between surfaces make
// long chains of rounds that a launch waits for: the 10,000-step walk of 1M spins
// on 2.56M triangles of overlapping tubes went 2.93e9 -> 3.56e9.
#pragma once
#include "common.cuh"
#include "engine.h"
#include "mesh_common.cuh"

namespace dsim {


static constexpr int kFlatThreads = 128;
static constexpr int kFlatWarps = kFlatThreads / 32;
static constexpr int kFlatSlots = 4;      // hits kept per owner per round
static constexpr uint32_t kFlatMaxWidth = 4;  // cells per axis of a box the warp handles

// A warp's lists
struct FlatLists {
    // the round's sub-segments by owner lane: start and excluded triangle
    // (bits); end - start and fine-cell box origin lo0 | lo1 << 10 | lo2 << 20
    // (bits)
    float4 o[32], d[32];
    uint32_t src[32];  // by rank among the lanes with cells (flat_box)
    uint2 cell[64];    // cells with records still to test: first record, owner | count << 5
    uint32_t n[32];    // hits filed per owner
};

// Hits filed by owner.  FlatWarp keeps a hit as its triangle and the fraction r
// of the sub-segment with two flags in its top bits (0 < r < 1 leaves them
// free), and works the point and its distance out again, by the test's own
// expressions, for the hit it wants: 1 KB a warp instead of 3, which is L1 that
// a step's records can stay in.  HitWarp keeps all of a hit, for the forms whose
// points come by other ways.
struct FlatWarp : FlatLists {
    uint32_t t[kFlatSlots][32];
    uint32_t r[kFlatSlots][32];
};
struct HitWarp : FlatLists {
    uint32_t t[kFlatSlots][32];
    uint32_t type[kFlatSlots][32];
    float d2[kFlatSlots][32];
    float x[kFlatSlots][32];
    float y[kFlatSlots][32];
    float z[kFlatSlots][32];
};

__device__ __forceinline__ void file_hit(FlatWarp& H, uint32_t owner, const FastHit& h) {
    const uint32_t slot = atomicAdd(&H.n[owner], 1u);
    if (slot < (uint32_t)kFlatSlots) {
        H.t[slot][owner] = h.t;
        H.r[slot][owner] = __float_as_uint(h.r) | ((h.type & kHitWalk) ? 0x80000000u : 0u) |
                           ((h.type & ~kHitWalk) > 1u ? 0x40000000u : 0u);
    }
}
__device__ __forceinline__ void file_hit(HitWarp& H, uint32_t owner, const FastHit& h) {
    uint32_t slot = atomicAdd(&H.n[owner], 1u);
    if (slot < (uint32_t)kFlatSlots) {
        H.t[slot][owner] = h.t; H.type[slot][owner] = h.type; H.d2[slot][owner] = h.d2;
        H.x[slot][owner] = h.x; H.y[slot][owner] = h.y; H.z[slot][owner] = h.z;
    }
}
// the lane's own hit q (without its walk flag; an edge's and a vertex's type
// count the same), and whether it has that flag
__device__ __forceinline__ FastHit filed_hit(const FlatWarp& H, uint32_t q, uint32_t lane) {
    const uint32_t bits = H.r[q][lane];
    const float4 O = H.o[lane], D = H.d[lane];
    FastHit h;
    h.t = H.t[q][lane];
    h.type = 1u + ((bits >> 30) & 1u);
    h.r = __uint_as_float(bits & 0x3FFFFFFFu);
    h.x = O.x + D.x * h.r; h.y = O.y + D.y * h.r; h.z = O.z + D.z * h.r;
    h.d2 = (O.x - h.x) * (O.x - h.x) + (O.y - h.y) * (O.y - h.y) + (O.z - h.z) * (O.z - h.z);
    return h;
}
__device__ __forceinline__ bool filed_walk(const FlatWarp& H, uint32_t q, uint32_t lane) { return H.r[q][lane] >> 31; }
__device__ __forceinline__ FastHit filed_hit(const HitWarp& H, uint32_t q, uint32_t lane) {
    FastHit h;
    h.t = H.t[q][lane]; h.type = H.type[q][lane] & ~kHitWalk; h.d2 = H.d2[q][lane]; h.r = 0.0f;
    h.x = H.x[q][lane]; h.y = H.y[q][lane]; h.z = H.z[q][lane];
    return h;
}
__device__ __forceinline__ bool filed_walk(const HitWarp& H, uint32_t q, uint32_t lane) {
    return H.type[q][lane] & kHitWalk;
}

// A lane's state that only the ends of steps and the hits read, kept in shared
// memory: a round's lists and tests hold nearly every register, and what does
// not fit is spilled around them.  In the plain step these words take the form
// of 7 blocks per SM from 204 B of spills to 32 and make it the fastest over
// many waves (us per step at 4 / 5 / 6 / 7 / 8 / 9 blocks per SM: 400,000 spins
// on 100 tubes 46.6 / 40.8 / 39.0 / 37.0 / 38.7 / 41.7, 1M spins on 400 tubes
// 119.4 / 103.0 / 98.3 / 97.8 / 98.5 / 102.4; in registers, at 5: 41.7 and
// 105.6).
struct LaneState {
    float mag[32], umax[32], umin[32], u[32];
    uint32_t comp[32], fiber[32], nrefl[32], nperm[32], status[32], it[32], sub[32];
};

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v, uint32_t lane) {
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1) {
        uint32_t t = __shfl_up_sync(0xFFFFFFFFu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

// ---- flat lists over the warp -----------------------------------------------
// Lane k's `count` elements (none or more) occupy [start, start + count) of a
// flat list.  For the 32 elements from `base` on, the warp's starts among them
// form one mask (a hardware OR-reduction), and element base + l belongs to the
// lane whose rank among the lanes with elements is the number of starts up to
// it, less one; a table in shared memory takes the rank to the lane.  A binary
// search of the prefix sums by shuffles took five dependent shuffles instead.
__device__ __forceinline__ uint32_t flat_starts(bool has, uint32_t start, uint32_t base) {
    const uint32_t k = start - base;
    return __reduce_or_sync(0xFFFFFFFFu, (has && k < 32u) ? 1u << k : 0u);
}

// A lane's fine-cell box, from absolute end points: its cells are counted with
// the y and z widths rounded up to 1, 2 or 4 (so an element's cell needs no
// division; the cells beyond the box are skipped).  Boxes wider than 4 cells
// are left to their owner (solo).
struct FlatBox {
    uint32_t lo0, lo1, lo2, w0, w1, w2, count, packed;
    bool solo;
};
__device__ __forceinline__ FlatBox flat_box(const AccelDev& acc, bool open, float ox, float oy, float oz, float px,
                                            float py, float pz) {
    FlatBox b;
    b.lo0 = b.lo1 = b.lo2 = b.w0 = b.w1 = b.w2 = b.count = b.packed = 0;
    b.solo = false;
    if (open) {
        const float invLf = acc.invLf;
        const uint32_t nf = acc.nf;
        b.lo0 = fine_coord(fminf(ox, px) - kAccelEps, invLf, nf);
        b.lo1 = fine_coord(fminf(oy, py) - kAccelEps, invLf, nf);
        b.lo2 = fine_coord(fminf(oz, pz) - kAccelEps, invLf, nf);
        b.w0 = fine_coord(fmaxf(ox, px) + kAccelEps, invLf, nf) - b.lo0 + 1;
        b.w1 = fine_coord(fmaxf(oy, py) + kAccelEps, invLf, nf) - b.lo1 + 1;
        b.w2 = fine_coord(fmaxf(oz, pz) + kAccelEps, invLf, nf) - b.lo2 + 1;
        b.solo = max(b.w0, max(b.w1, b.w2)) > kFlatMaxWidth;
        const uint32_t b2 = (b.w2 > 1u) + (b.w2 > 2u), b12 = b2 + (b.w1 > 1u) + (b.w1 > 2u);
        if (!b.solo) {
            b.count = b.w0 << b12;
            b.packed = (b2 << 5) | (b12 << 7) | ((b.w1 - 1u) << 10) | ((b.w2 - 1u) << 12);
        }
    }
    return b;
}

// fills the rank table of the lanes' boxes; returns the elements in all.  first:
// the lane's first element
__device__ __forceinline__ uint32_t flat_items(FlatLists& H, const FlatBox& b, uint32_t lane, uint32_t& first) {
    const uint32_t incl = warp_incl_scan(b.count, lane);
    first = incl - b.count;
    const uint32_t some = __ballot_sync(0xFFFFFFFFu, b.count > 0);
    if (b.count > 0) H.src[__popc(some & ((1u << lane) - 1u))] = lane | b.packed | (first << 14);
    return __shfl_sync(0xFFFFFFFFu, incl, 31);
}

// element m's owner and cell offset in its box; false beyond the box
__device__ __forceinline__ bool flat_cell(uint32_t src, uint32_t m, uint32_t& ow, uint32_t& ix, uint32_t& iy,
                                          uint32_t& iz) {
    const uint32_t q = m - (src >> 14), b2 = (src >> 5) & 3u, b12 = (src >> 7) & 7u;
    ow = src & 31u;
    ix = q >> b12;
    iy = (q & ((1u << b12) - 1u)) >> b2;
    iz = q & ((1u << b2) - 1u);
    return (iy <= ((src >> 10) & 3u)) & (iz <= ((src >> 12) & 3u));
}

// The round's records, window by window (one per warp; the members are
// warp-uniform but for first, cells, start, cnt and b0).  Cells are looked up 32
// at a time (flat_cell, cell_records); those with records left wait in H.cell
// until 32 of them (or the last) make a block, whose records form one flat
// list: so windows are full but for a block's last.
struct FlatList {
    uint32_t itotal, first, cells;  // elements in all; the lane's first one and their number
    uint32_t ib, before;            // next element; boxes begun before it
    uint32_t nq;                    // cells waiting
    uint32_t rb, total, from;       // next record of the block, records in it, its cells begun before rb
    uint32_t start, cnt, b0;        // lane's cell of the block: first record in the flat list, count, record index
};
__device__ __forceinline__ FlatList flat_list(FlatLists& H, const FlatBox& b, uint32_t lane) {
    FlatList l;
    l.cells = b.count;
    l.itotal = flat_items(H, b, lane, l.first);
    l.ib = l.before = l.nq = l.rb = l.total = l.from = l.start = l.cnt = l.b0 = 0;
    return l;
}
// Makes the next block when the current one's records are used up; false when
// no record is left.  at(owner, O): the owner's absolute start.
template <class At>
__device__ __forceinline__ bool flat_next(FlatLists& H, FlatList& l, const AccelDev& acc, uint32_t lane, At at) {
    const uint32_t below = (1u << lane) - 1u;
    while (l.rb >= l.total && (l.ib < l.itotal || l.nq > 0)) {
        if (l.ib < l.itotal && l.nq < 32) {
            const uint32_t begun = flat_starts(l.cells > 0, l.first, l.ib);
            const uint32_t src = H.src[l.before + __popc(begun & (below * 2u + 1u)) - 1u];
            l.before += __popc(begun);
            uint32_t b0 = 0, cnt = 0, ow, ix, iy, iz;
            if (flat_cell(src, l.ib + lane, ow, ix, iy, iz) && l.ib + lane < l.itotal) {
                const float4 D = H.d[ow];
                const float4 O = at(ow, H.o[ow]);
                const uint32_t bx = __float_as_uint(D.w);
                cell_records(acc, (bx & 1023u) + ix, ((bx >> 10) & 1023u) + iy, (bx >> 20) + iz, O.x, O.y, O.z, D.x,
                             D.y, D.z, b0, cnt);
            }
            const uint32_t some = __ballot_sync(0xFFFFFFFFu, cnt > 0);
            if (cnt > 0) H.cell[l.nq + __popc(some & below)] = make_uint2(b0, ow | (cnt << 5));
            l.nq += __popc(some);
            l.ib += 32;
            __syncwarp();
        } else {
            const uint32_t k = min(l.nq, 32u);
            l.nq -= k;
            const uint2 c = lane < k ? H.cell[l.nq + lane] : make_uint2(0u, 0u);
            l.b0 = c.x;
            l.cnt = c.y >> 5;
            const uint32_t incl = warp_incl_scan(l.cnt, lane);
            l.start = incl - l.cnt;
            l.total = __shfl_sync(0xFFFFFFFFu, incl, 31);
            l.rb = l.from = 0;
            if (lane < k) H.cell[l.nq + lane] = make_uint2(c.x - l.start, c.y & 31u);  // record - flat index, owner
            __syncwarp();
        }
    }
    return l.rb < l.total;
}
// record e and owner o of flat record base + lane (call in ascending order of
// base; all lanes; meaningless past the block's total)
__device__ __forceinline__ void flat_pick(const FlatLists& H, FlatList& l, uint32_t lane, uint32_t base, uint32_t& e,
                                          uint32_t& o) {
    const uint32_t begun = flat_starts(l.cnt > 0, l.start, base);
    const uint2 c = H.cell[l.nq + l.from + __popc(begun & (0xFFFFFFFFu >> (31u - lane))) - 1u];
    l.from += __popc(begun);
    e = c.x + base + lane;
    o = c.y;
}

// Queue of a warp's 32-byte records that passed the plane test, as (record,
// owner) pairs: the rest of the exact test (with its dependent loads) runs on
// 32 of them at a time with every lane busy
static constexpr uint32_t kFlatQueue = 96;  // at most 31 left over + a window of 64
struct FlatQueue {
    uint2 eo[kFlatQueue];
};

// one 32-byte record already in registers against a sub-segment
__device__ __forceinline__ bool test_wide_loaded(const MeshDev& g, float4 q, float4 pt, float4 O, float4 D,
                                                 FastHit& h) {
    if (!plane_may_cross(q, O.x, O.y, O.z, D.x, D.y, D.z)) return false;
    if (__float_as_uint(pt.w) == __float_as_uint(O.w)) return false;
    return test_split(g, q, pt, O.x, O.y, O.z, D.x, D.y, D.z, h);
}

// Staging of 32-byte records in shared memory by bulk copies (the TMA engine,
// cp.async.bulk): the records of a round's cells are taken in windows of 64;
// for each window, every lane whose cell overlaps it issues one bulk copy of
// its part (each cell's records are contiguous), completing on the warp's
// mbarrier, whose expected byte count lane 0 posts first.  Two buffers: the
// next window's copies are in flight while the current one is tested.  Waits
// are bounded: past kStageSpinLimit polls the warp records kStatusStageTimeout
// and stops stepping (its spins are not written back).
static constexpr uint32_t kStageRecs = 64;
static constexpr uint32_t kStageSpinLimit = 1u << 20;
struct __align__(128) FlatStage {
    float4 rec[2][kStageRecs][2];  // [buffer][record][q, pt]
    unsigned long long bar[2];     // one mbarrier per buffer
    uint32_t parity[2];            // the phase each buffer waits for next
    uint32_t abort;                // a wait ran out
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// lane 0 of a warp, once per kernel (before any copy)
__device__ __forceinline__ void stage_init(FlatStage* P) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&P->bar[0])) : "memory");
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&P->bar[1])) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    P->parity[0] = P->parity[1] = 0u;
    P->abort = 0u;
}

// lane 0: the window's total bytes, posted before the copies are issued
__device__ __forceinline__ void stage_expect(FlatStage* P, uint32_t buf, uint32_t bytes) {
    asm volatile("{\n .reg .b64 st;\n mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n}\n"
                 ::"r"(smem_u32(&P->bar[buf])), "r"(bytes) : "memory");
}

// one bulk copy of n 32-byte records (16-byte aligned source and destination)
__device__ __forceinline__ void stage_copy(FlatStage* P, uint32_t buf, uint32_t at, const AccelRecWide* src,
                                           uint32_t n) {
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");  // the buffer's earlier generic reads first
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
            smem_u32(&P->rec[buf][at][0])),
        "l"(src), "r"(n * 32u), "r"(smem_u32(&P->bar[buf]))
        : "memory");
}

// every lane: wait for the buffer's copies (bounded); false when it timed out
__device__ __forceinline__ bool stage_wait(FlatStage* P, uint32_t buf) {
    const uint32_t bar = smem_u32(&P->bar[buf]), par = P->parity[buf];
    uint32_t done = 0;
    for (uint32_t k = 0; k < kStageSpinLimit && !done; k++) {
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done)
            : "r"(bar), "r"(par)
            : "memory");
    }
    __syncwarp();
    return __all_sync(0xFFFFFFFFu, done != 0u);
}

// the rest of the exact test of queued record e for owner o (plane test passed)
__device__ __forceinline__ void flat_test_queued(FlatWarp& H, const MeshDev& g, const AccelDev& acc, uint32_t e,
                                                 uint32_t o) {
    const float4 q = __ldg(&acc.recw[e].q), pt = __ldg(&acc.recw[e].pt);
    const float4 O = H.o[o], D = H.d[o];
    FastHit h;
    if (__float_as_uint(pt.w) != __float_as_uint(O.w) && test_split(g, q, pt, O.x, O.y, O.z, D.x, D.y, D.z, h))
        file_hit(H, o, h);
}

// appends the lanes' surviving pairs to the queue (qn: warp-uniform length) and
// tests full groups of 32 from its top, with `last` (warp-uniform) the partial
// group too: one copy of the exact test a round
__device__ __forceinline__ void flat_enqueue(FlatWarp& H, FlatQueue& Q, const MeshDev& g, const AccelDev& acc,
                                             uint32_t lane, bool s0, uint32_t e0, uint32_t o0, bool s1, uint32_t e1,
                                             uint32_t o1, uint32_t& qn, bool last) {
    const uint32_t b0 = __ballot_sync(0xFFFFFFFFu, s0), b1 = __ballot_sync(0xFFFFFFFFu, s1);
    const uint32_t below = (1u << lane) - 1u;
    if (s0) Q.eo[qn + __popc(b0 & below)] = make_uint2(e0, o0);
    qn += __popc(b0);
    if (s1) Q.eo[qn + __popc(b1 & below)] = make_uint2(e1, o1);
    qn += __popc(b1);
    __syncwarp();
    while (qn >= 32 || (last && qn > 0)) {
        const uint32_t k = min(qn, 32u);
        qn -= k;
        if (lane < k) flat_test_queued(H, g, acc, Q.eo[qn + lane].x, Q.eo[qn + lane].y);
        __syncwarp();
    }
}

// A lane whose box is too wide for the warp's list: its own records, cell by
// cell (rare, and out of line so that the box's corners need not be kept)
static __device__ __noinline__ void flat_solo(FlatWarp& H, const MeshDev& g, const AccelDev& acc, uint32_t lane,
                                              float px, float py, float pz) {
    const float4 O = H.o[lane], D = H.d[lane];
    const FlatBox b = flat_box(acc, true, O.x, O.y, O.z, px, py, pz);
    for (uint32_t ix = 0; ix < b.w0; ix++)
        for (uint32_t iy = 0; iy < b.w1; iy++)
            for (uint32_t iz = 0; iz < b.w2; iz++) {
                const uint32_t key = morton3(b.lo0 + ix, b.lo1 + iy, b.lo2 + iz);
                const uint32_t b0 = __ldg(acc.start + key), b1 = __ldg(acc.start + key + 1);
                for (uint32_t k = b0; k < b1; k++) {
                    FastHit h;
                    if (test_entry(g, acc, k, __float_as_uint(O.w), O.x, O.y, O.z, D.x, D.y, D.z, h))
                        file_hit(H, lane, h);
                }
            }
}

// Are the lane's n filed hits one hit (filed once per fine cell that lists its
// triangle), at (x, y, z), that needs no walk?  Then it is the reference's.
template <class Hits>
__device__ __forceinline__ bool flat_only_hit(const Hits& H, uint32_t lane, uint32_t n, uint32_t gn, float x, float y,
                                              float z) {
    const uint32_t t = H.t[0][lane];
    bool one = n <= (uint32_t)kFlatSlots && !filed_walk(H, 0, lane);
    if (n > 1) one = one && H.t[1][lane] == t && (n < 3 || H.t[2][lane] == t) && (n < 4 || H.t[3][lane] == t);
    const float inv = 0.5f * (float)gn, margin = 2.0f * kRegularEps * inv;
    return one & clear_of_faces(x, inv, margin) & clear_of_faces(y, inv, margin) & clear_of_faces(z, inv, margin);
}
// The slot of the reference's hit among several (n <= kFlatSlots) by the walk
// over its cells, kNoPlace for none.  About one hit in ten needs it: out of
// line, so that a round keeps neither its registers nor its code.
template <class Hits>
static __device__ __noinline__ uint32_t flat_choose(const Hits& H, const MeshDev& g, uint32_t lane, uint32_t n,
                                                    RefWalk w) {
    uint32_t bq = kNoPlace, bt = 0, bplace = kNoPlace;
    float bd2 = 0.0f;
    for (uint32_t q = 0; q < n; q++) {
        const uint32_t t = H.t[q][lane];
        if (bq != kNoPlace && t == bt) continue;  // filed from another fine cell too
        const uint32_t place = first_place(g, w, __ldg(g.tri_cells + t), t);
        if (place == kNoPlace) continue;
        const float d2 = filed_hit(H, q, lane).d2;
        if (place < bplace || (place == bplace && (d2 < bd2 || (d2 == bd2 && t < bt)))) {
            bq = q; bplace = place; bt = t; bd2 = d2;
        }
    }
    return bq;
}

// One round for every lane of the warp (all 32 lanes call it).  open: the lane
// has a sub-segment (o -> p, `excluded` = last-hit triangle) to test.  On
// return, for open lanes, found / best hold the reference's collision result
// (its FP32 tests).  LAYOUT: 1 or 2 compile only the 32- or 64-byte record
// path; 0 dispatches on acc.wide at run time (every layout).  Q (32-byte
// records only): records past the plane test are queued and finished 32 at a
// time (null: finished in place)
template <int LAYOUT = 0>
__device__ __forceinline__ void flat_round_mode(FlatWarp& H, const MeshDev& g, const AccelDev& acc,
                                                uint32_t lane, bool open, float ox, float oy, float oz,
                                                float px, float py, float pz, uint32_t excluded,
                                                bool& found, FastHit& best, FlatQueue* Q = nullptr,
                                                FlatStage* P = nullptr) {
    const float dx = px - ox, dy = py - oy, dz = pz - oz;
    const FlatBox box = flat_box(acc, open, ox, oy, oz, px, py, pz);
    H.o[lane] = make_float4(ox, oy, oz, __uint_as_float(excluded));
    H.d[lane] = make_float4(dx, dy, dz, __uint_as_float(box.lo0 | (box.lo1 << 10) | (box.lo2 << 20)));
    H.n[lane] = 0;
    FlatList l = flat_list(H, box, lane);
    __syncwarp();
    auto at = [](uint32_t, float4 O) { return O; };
    if (LAYOUT == 1 && Q) {
        // records past the plane test are queued and finished 32 at a time
        uint32_t qn = 0;
        for (;;) {
            const bool more = flat_next(H, l, acc, lane, at);  // warp-uniform
            bool s0 = false, s1 = false;
            uint32_t e0 = 0, e1 = 0, o0 = 0, o1 = 0;
            if (more) {
                flat_pick(H, l, lane, l.rb, e0, o0);
                flat_pick(H, l, lane, l.rb + 32, e1, o1);
                s0 = l.rb + lane < l.total;
                s1 = l.rb + 32 + lane < l.total;
                float4 q0 = make_float4(0.f, 0.f, 0.f, 0.f), q1 = q0;
                if (s0) q0 = __ldg(&acc.recw[e0].q);
                if (s1) q1 = __ldg(&acc.recw[e1].q);
                if (s0) {
                    const float4 O = H.o[o0], D = H.d[o0];
                    s0 = plane_may_cross(q0, O.x, O.y, O.z, D.x, D.y, D.z);
                }
                if (s1) {
                    const float4 O = H.o[o1], D = H.d[o1];
                    s1 = plane_may_cross(q1, O.x, O.y, O.z, D.x, D.y, D.z);
                }
                l.rb += 64;
            }
            flat_enqueue(H, *Q, g, acc, lane, s0, e0, o0, s1, e1, o1, qn, !more);
            if (!more) break;
        }
    } else if (LAYOUT == 1 && P) {
        while (flat_next(H, l, acc, lane, at)) {
            // windows of kStageRecs records staged by bulk copies, the next one in
            // flight while this one is tested
            const uint32_t nwin = (l.total + kStageRecs - 1) / kStageRecs;
            auto issue = [&](uint32_t w, uint32_t buf) {
                const uint32_t lo = w * kStageRecs, hi = min(lo + kStageRecs, l.total);
                if (lane == 0) stage_expect(P, buf, (hi - lo) * 32u);
                __syncwarp();
                const uint32_t a = max(l.start, lo), z = min(l.start + l.cnt, hi);
                if (a < z) stage_copy(P, buf, a - lo, acc.recw + l.b0 + (a - l.start), z - a);
            };
            if (!P->abort) issue(0, 0);
            for (uint32_t w = 0; w < nwin && !P->abort; w++) {
                const uint32_t buf = w & 1u;
                if (w + 1 < nwin) issue(w + 1, buf ^ 1u);
                if (!stage_wait(P, buf)) {
                    // a wait ran out: wait once more (bounded) for the copies in
                    // flight to this buffer and the next, then stop the warp
                    stage_wait(P, buf);
                    if (w + 1 < nwin) stage_wait(P, buf ^ 1u);
                    if (lane == 0) P->abort = 1u;
                    __syncwarp();
                    break;
                }
                if (lane == 0) P->parity[buf] ^= 1u;
#pragma unroll
                for (uint32_t half = 0; half < 64; half += 32) {
                    const uint32_t at0 = w * kStageRecs + half;
                    uint32_t e, o;
                    flat_pick(H, l, lane, at0, e, o);
                    FastHit h;
                    if (at0 + lane < l.total && test_wide_loaded(g, P->rec[buf][half + lane][0],
                                                                 P->rec[buf][half + lane][1], H.o[o], H.d[o], h))
                        file_hit(H, o, h);
                }
                __syncwarp();  // the buffer's reads end before its next copies
            }
            l.rb = l.total;
        }
    } else {
        // tested in place
        while (flat_next(H, l, acc, lane, at)) {
            uint32_t e, o;
            flat_pick(H, l, lane, l.rb, e, o);
            if (l.rb + lane < l.total) {
                const float4 O = H.o[o], D = H.d[o];
                const uint32_t excl = __float_as_uint(O.w);
                FastHit h;
                bool hit;
                if (LAYOUT == 2 || (LAYOUT == 0 && acc.wide == 2))
                    hit = test_full(load_full(acc.recf + e), excl, O.x, O.y, O.z, D.x, D.y, D.z, h);
                else if (LAYOUT == 1 || acc.wide == 1)
                    hit = test_wide_loaded(g, __ldg(&acc.recw[e].q), __ldg(&acc.recw[e].pt), O, D, h);
                else
                    hit = test_narrow(g, acc, e, excl, O.x, O.y, O.z, D.x, D.y, D.z, h);
                if (hit) file_hit(H, o, h);
            }
            l.rb += 32;
            __syncwarp();
        }
    }
    // wider boxes (long sub-segments): the owner alone
    if (box.solo) flat_solo(H, g, acc, lane, px, py, pz);
    __syncwarp();
    found = false;
    if (!open) return;
    const uint32_t n = H.n[lane];
    if (n == 0) return;
    found = true;
    best = filed_hit(H, 0, lane);
    if (!flat_only_hit(H, lane, n, g.n, best.x, best.y, best.z)) {
        if (n > (uint32_t)kFlatSlots) {
            FastHit h;  // (best itself stays in registers)
            bool any;
            ref_scan(g, ox, oy, oz, px, py, pz, excluded, h, any);
            found = any;
            if (any) best = h;
            return;
        }
        const uint32_t gn = g.n;
        const float L = g.L;
        const uint32_t bq =
            flat_choose(H, g, lane, n,
                        ref_walk(ref_coord(ox, L, gn), ref_coord(oy, L, gn), ref_coord(oz, L, gn),
                                 ref_coord(px, L, gn), ref_coord(py, L, gn), ref_coord(pz, L, gn)));
        found = bq != kNoPlace;
        if (found) best = filed_hit(H, bq, lane);
    }
}

// Reflection or permeation at the round's hit `best`: the permeation interval
// [umin, umax], the compartment transition table and the mirror reflection
// of dSim3/src/spinKernelCpu.cpp:238-271 and :406-422; the hit point becomes
// the next sub-segment's start and its triangle the excluded one.
__device__ __forceinline__ void apply_hit(const MeshDev& g, const FastHit& best, float u, float perm,
                                          uint32_t reflType, float& umax, float& umin, float& ox,
                                          float& oy, float& oz, float& px, float& py, float& pz,
                                          uint32_t& comp, uint32_t& fiber, uint32_t& excluded,
                                          uint32_t& nrefl, uint32_t& nperm) {
    float thr = umax - (umax - umin) * perm;
    if (u <= thr) {
        if ((reflType == 0) | (best.type > 1)) {
            px = ox; py = oy; pz = oz;
        } else {
            const float4 nn = __ldg(reinterpret_cast<const float4*>(g.plane + best.t));
            float nx = nn.x, ny = nn.y, nz = nn.z;
            float sx2 = px - best.x, sy2 = py - best.y, sz2 = pz - best.z;
            px = (1.0f - 2.0f * nx * nx) * sx2 - 2.0f * nx * ny * sy2 - 2.0f * nx * nz * sz2 + best.x;
            py = -2.0f * nx * ny * sx2 + (1.0f - 2.0f * ny * ny) * sy2 - 2.0f * ny * nz * sz2 + best.y;
            pz = -2.0f * nx * nz * sx2 - 2.0f * ny * nz * sy2 + (1.0f - 2.0f * nz * nz) * sz2 + best.z;
        }
        umax = thr;
        nrefl++;
    } else {
        umin = thr;
        nperm++;
        uint32_t info = __ldg(&g.plane[best.t].info);
        uint32_t membrane = info & 3u;
        if (comp == 2) {
            if (membrane == 0) comp = 1;
            else { comp = 0; fiber = 0xFFFFu; }
        } else if (comp == 1) {
            comp = 2;
        } else if (comp == 3) {
            comp = 0; fiber = 0xFFFFu;
        } else {
            fiber = (info >> 2) & 0xFFFFu;
            comp = (membrane == 1) ? 2u : 3u;
        }
    }
    ox = best.x; oy = best.y; oz = best.z;
    excluded = best.t;
}

}  // namespace dsim
