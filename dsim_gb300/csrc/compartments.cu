// compartments.cu -- which compartment and fiber each spin starts in (GPU).
//
// Reference: SpinSystem::findSpinsInFibers, dSim3/src/spinSystem.cpp:1615-1852.
// A line is drawn from the spin out of the volume along the axis of its
// largest coordinate, to 1.1 times the mesh extent on that axis
// (spinSystem.cpp:1676-1684).  A closed membrane encloses the spin when the
// line crosses it an odd number of times; membranes are examined innermost
// type first (axon 0, myelin 1, glia 2), giving compartment 1, 2 or 3, else 0
// (outside).  If the line touches a triangle edge or vertex the answer is
// ambiguous and the line is tilted by a random offset of up to 0.05 per axis
// and tried again (:1686-1692); after 20 failed tries the spin is moved to a
// random position and examined anew (:1659-1665).
//
// Here the line is followed through the fine acceleration grid, by a warp or by a
// thread (launch_compartments), with the same result.  A crossing is counted only
// in the cell that contains the crossing point, so a triangle listed in several
// cells counts once.  Crossing parity is kept per (fiber, membrane).
// The reference takes its candidates from an R-tree in tree order; when two
// fibers of the same membrane type both enclose a spin (overlapping meshes)
// it keeps the last one in that order, while these kernels keep the lowest
// fiber index.  For meshes without overlaps the result is the same.
// Tilts and moves draw from Philox keyed by the caller's seed and the spin.
#include <cmath>
#include "common.cuh"
#include "engine.h"
#include "mesh_common.cuh"

namespace dsim {

static constexpr int kParitySlots = 32;

__device__ __forceinline__ float sgn_ref(float v) { return (v >= 0.0f) ? 1.0f : -1.0f; }

struct Point {
    float x, y, z;
};
// spinSystem.cpp:1659-1665: a new random position in the start box
__device__ __forceinline__ Point new_place(uint32_t id, uint32_t move, float startBox, uint32_t key0, uint32_t key1) {
    const u32x4 r = philox4x32_10({id, move, 0u, 0xB0C5u}, key0, key1);
    return {startBox * 2.0f * ((float)(r.x >> 8) * 0x1p-24f - 0.5f),
            startBox * 2.0f * ((float)(r.y >> 8) * 0x1p-24f - 0.5f),
            startBox * 2.0f * ((float)(r.z >> 8) * 0x1p-24f - 0.5f)};
}
// the end of try tr's line from s, tilted from the second try on
__device__ __forceinline__ Point line_end(Point s, float mx, float my, float mz, uint32_t id, uint32_t tr,
                                          uint32_t move, uint32_t key0, uint32_t key1) {
    Point e = s;
    const float ax = fabsf(s.x), ay = fabsf(s.y), az = fabsf(s.z);
    if ((ax > ay) & (ax > az)) e.x = (float)((double)sgn_ref(s.x) * 1.1 * (double)mx);
    else if (ay > az) e.y = (float)((double)sgn_ref(s.y) * 1.1 * (double)my);
    else e.z = (float)((double)sgn_ref(s.z) * 1.1 * (double)mz);
    if (tr > 0) {
        const u32x4 r = philox4x32_10({id, tr, move, 0xC0A5u}, key0, key1);
        e.x = (float)((double)e.x + (double)((float)(r.x >> 8) * 0x1p-24f) * 0.05);
        e.y = (float)((double)e.y + (double)((float)(r.y >> 8) * 0x1p-24f) * 0.05);
        e.z = (float)((double)e.z + (double)((float)(r.z >> 8) * 0x1p-24f) * 0.05);
    }
    return e;
}

// ---- a warp per spin ------------------------------------------------------------
// Lane l takes the layers l, l + 32, ... of cells across the line's main axis,
// looks up the cells the line passes there and tests the records of those whose
// slab it may meet; lane s holds entry s of the parity list.  Bound by the latency
// of the dependent loads (cell, record, triangle), of which a thread has a hundred
// layers' in turn: 100,001 spins on 640,000 triangles 1.22 -> 0.58 ms.
//
// a lane's walk over its share of the line's cells and their records
struct LineWalk {
    uint32_t ca, cb, cc, lob, hib, loc, hic;  // layer, cell in it and the layer's range
    uint32_t k, end;                          // records of the cell
};

__global__ void __launch_bounds__(128) k_compartments_warp(MeshDev g, AccelDev acc, SpinsSorted S, float mx, float my,
                                                      float mz, float startBox, uint32_t key0, uint32_t key1,
                                                      uint32_t maxTries, uint32_t maxMoves, uint32_t* status,
                                                      uint32_t* moved) {
    const uint32_t FULL = 0xFFFFFFFFu, lane = threadIdx.x & 31u;
    // warp-uniform, as all but the walk; the threads of all spins' warps pass 2^32 from 2^27 spins on
    const uint32_t i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (i >= S.N) return;
    float sx = S.x[i], sy = S.y[i], sz = S.z[i];
    const uint32_t id = S.id[i];
    const uint32_t nf = acc.nf;
    const float cell = 1.0f / acc.invLf;
    bool resolved = false;
    uint32_t comp = 0, fiber = 0xFFFFu, st = 0, nMoves = 0;
    for (uint32_t move = 0; move <= maxMoves && !resolved; move++) {
        if (move > 0) {
            const Point p = new_place(id, move, startBox, key0, key1);
            sx = p.x; sy = p.y; sz = p.z;
            nMoves++;
        }
        for (uint32_t tr = 0; tr <= maxTries && !resolved; tr++) {
            const Point e = line_end({sx, sy, sz}, mx, my, mz, id, tr, move, key0, key1);
            const float ex = e.x, ey = e.y, ez = e.z;
            const float dx = ex - sx, dy = ey - sy, dz = ez - sz;
            // main axis m0, the other two m1 < m2
            const int m0 = (fabsf(dx) >= fabsf(dy) && fabsf(dx) >= fabsf(dz)) ? 0 : (fabsf(dy) >= fabsf(dz) ? 1 : 2);
            const float pa = m0 == 0 ? sx : (m0 == 1 ? sy : sz), da = m0 == 0 ? dx : (m0 == 1 ? dy : dz);
            const float pb = m0 == 0 ? sy : sx, db = m0 == 0 ? dy : dx;
            const float pc = m0 == 2 ? sy : sz, dc = m0 == 2 ? dy : dz;
            const uint32_t lo = fine_coord(fminf(pa, pa + da) - kAccelEps, acc.invLf, nf);
            const uint32_t hi = fine_coord(fmaxf(pa, pa + da) + kAccelEps, acc.invLf, nf);
            const float inv = 1.0f / da;
            uint32_t key = 0, nkeys = 0, parity = 0;  // lane s: entry s of the list
            uint32_t edgeTypes = 0;  // membrane types whose triangles were met at an edge or vertex
            LineWalk w;
            w.ca = lo + lane;
            w.cb = 1; w.hib = 0;  // past the end of a layer
            w.cc = w.loc = w.hic = w.lob = 0;
            w.k = w.end = 0;
            bool started = false;
            for (;;) {
                // the lane's next record
                while (w.k >= w.end && w.ca <= hi) {
                    if (started) {
                        if (w.cc < w.hic) w.cc++;
                        else { w.cc = w.loc; w.cb++; }
                    }
                    if (!started || w.cb > w.hib) {
                        if (started) w.ca += 32;
                        started = true;
                        if (w.ca > hi) break;
                        // the cells the layer's part of the line passes, the layer
                        // and the line widened by kAccelEps and more than the
                        // rounding here (under 2e-6); the outermost layers are open
                        float t0 = (-1.0f + (float)w.ca * cell - 2.0f * kAccelEps - pa) * inv;
                        float t1 = (-1.0f + (float)(w.ca + 1) * cell + 2.0f * kAccelEps - pa) * inv;
                        if (w.ca == 0) t0 = da > 0.0f ? 0.0f : 1.0f;
                        if (w.ca == nf - 1) t1 = da > 0.0f ? 1.0f : 0.0f;
                        t0 = fminf(fmaxf(t0, 0.0f), 1.0f);
                        t1 = fminf(fmaxf(t1, 0.0f), 1.0f);
                        const float b0f = pb + t0 * db, b1f = pb + t1 * db, c0f = pc + t0 * dc, c1f = pc + t1 * dc;
                        w.lob = fine_coord(fminf(b0f, b1f) - kAccelEps, acc.invLf, nf);
                        w.hib = fine_coord(fmaxf(b0f, b1f) + kAccelEps, acc.invLf, nf);
                        w.loc = fine_coord(fminf(c0f, c1f) - kAccelEps, acc.invLf, nf);
                        w.hic = fine_coord(fmaxf(c0f, c1f) + kAccelEps, acc.invLf, nf);
                        w.cb = w.lob;
                        w.cc = w.loc;
                    }
                    const uint32_t c0 = m0 == 0 ? w.ca : w.cb, c1 = m0 == 1 ? w.ca : (m0 == 0 ? w.cb : w.cc),
                                   c2 = m0 == 2 ? w.ca : w.cc;
                    uint32_t cnt;
                    cell_records(acc, c0, c1, c2, sx, sy, sz, dx, dy, dz, w.k, cnt);
                    w.end = w.k + cnt;
                }
                const bool live = w.k < w.end;
                if (!__any_sync(FULL, live)) break;
                bool hit = false;
                uint32_t fk = 0;  // fiber << 2 | membrane
                if (live) {
                    const uint32_t c0 = m0 == 0 ? w.ca : w.cb, c1 = m0 == 1 ? w.ca : (m0 == 0 ? w.cb : w.cc),
                                   c2 = m0 == 2 ? w.ca : w.cc;
                    FastHit h;
                    // count the crossing in the cell that holds it
                    if (test_entry(g, acc, w.k, 0xFFFFFFFFu, sx, sy, sz, dx, dy, dz, h) &&
                        fine_coord(h.x, acc.invLf, nf) == c0 && fine_coord(h.y, acc.invLf, nf) == c1 &&
                        fine_coord(h.z, acc.invLf, nf) == c2) {
                        hit = true;
                        fk = __ldg(&g.plane[h.t].info);
                        if ((h.type & ~kHitWalk) > 1) edgeTypes |= 1u << (fk & 3u);
                    }
                    w.k++;
                }
                for (uint32_t hits = __ballot_sync(FULL, hit); hits; hits &= hits - 1u) {
                    const uint32_t f = __shfl_sync(FULL, fk, __ffs(hits) - 1);
                    uint32_t at = __ballot_sync(FULL, lane < nkeys && key == f);
                    if (at == 0) {
                        if (nkeys == (uint32_t)kParitySlots) { st |= kStatusParityOverflow; continue; }
                        if (lane == nkeys) key = f;
                        at = 1u << nkeys++;
                    }
                    parity ^= at;
                }
            }
            edgeTypes = __reduce_or_sync(FULL, edgeTypes);
            uint32_t c = 0, f = 0xFFFFu, mt = 0;
            for (; mt < 3 && c == 0; mt++) {
                const uint32_t best = __reduce_min_sync(
                    FULL, (((parity >> lane) & 1u) && (key & 3u) == mt) ? key >> 2 : 0xFFFFFFFFu);
                if (best != 0xFFFFFFFFu) {
                    c = (mt == 0) ? 1u : ((mt == 2) ? 3u : 2u);
                    f = best & 0xFFFFu;
                }
            }
            // the membrane types examined (up to the one that encloses the spin)
            // must be free of edge and vertex crossings, as in the reference
            if (edgeTypes & ((1u << mt) - 1u)) continue;  // ambiguous: tilt the line and try again
            resolved = true;
            comp = c;
            fiber = f;
        }
    }
    if (lane != 0) return;
    if (!resolved) st |= kStatusUnresolved;
    S.x[i] = sx; S.y[i] = sy; S.z[i] = sz;
    S.meta[i] = (comp & 0xFFu) | (fiber << 8);
    if (nMoves) atomicAdd(moved, nMoves);
    if (st) atomicOr(status, st);
}

// ---- a thread per spin ----------------------------------------------------------
// Over every cell of the line's box: a third to two thirds of the warp's
// instructions, so the faster one where the spins fill the chip many times.
__global__ void __launch_bounds__(128) k_compartments_thread(MeshDev g, AccelDev acc, SpinsSorted S, float mx, float my,
                                                             float mz, float startBox, uint32_t key0, uint32_t key1,
                                                             uint32_t maxTries, uint32_t maxMoves, uint32_t* status,
                                                             uint32_t* moved) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= S.N) return;
    Point s = {S.x[i], S.y[i], S.z[i]};
    const uint32_t id = S.id[i];
    uint32_t keys[kParitySlots];
    uint32_t parity = 0, nkeys = 0;
    bool resolved = false;
    uint32_t comp = 0, fiber = 0xFFFFu, st = 0, nMoves = 0;
    for (uint32_t move = 0; move <= maxMoves && !resolved; move++) {
        if (move > 0) {
            s = new_place(id, move, startBox, key0, key1);
            nMoves++;
        }
        for (uint32_t tr = 0; tr <= maxTries && !resolved; tr++) {
            const Point e = line_end(s, mx, my, mz, id, tr, move, key0, key1);
            const float dx = e.x - s.x, dy = e.y - s.y, dz = e.z - s.z;
            const uint32_t lo0 = fine_coord(fminf(s.x, e.x) - kAccelEps, acc.invLf, acc.nf);
            const uint32_t lo1 = fine_coord(fminf(s.y, e.y) - kAccelEps, acc.invLf, acc.nf);
            const uint32_t lo2 = fine_coord(fminf(s.z, e.z) - kAccelEps, acc.invLf, acc.nf);
            const uint32_t hi0 = fine_coord(fmaxf(s.x, e.x) + kAccelEps, acc.invLf, acc.nf);
            const uint32_t hi1 = fine_coord(fmaxf(s.y, e.y) + kAccelEps, acc.invLf, acc.nf);
            const uint32_t hi2 = fine_coord(fmaxf(s.z, e.z) + kAccelEps, acc.invLf, acc.nf);
            nkeys = 0;
            parity = 0;
            uint32_t edgeTypes = 0;  // membrane types whose triangles were met at an edge or vertex
            for (uint32_t c2 = lo2; c2 <= hi2; c2++)
                for (uint32_t c1 = lo1; c1 <= hi1; c1++)
                    for (uint32_t c0 = lo0; c0 <= hi0; c0++) {
                        const uint32_t key = morton3(c0, c1, c2);
                        const uint32_t b0 = __ldg(acc.start + key), b1 = __ldg(acc.start + key + 1);
                        for (uint32_t k = b0; k < b1; k++) {
                            FastHit h;
                            if (!test_entry(g, acc, k, 0xFFFFFFFFu, s.x, s.y, s.z, dx, dy, dz, h)) continue;
                            // count the crossing in the cell that holds it
                            if (fine_coord(h.x, acc.invLf, acc.nf) != c0 || fine_coord(h.y, acc.invLf, acc.nf) != c1 ||
                                fine_coord(h.z, acc.invLf, acc.nf) != c2)
                                continue;
                            const uint32_t fk = __ldg(&g.plane[h.t].info);  // fiber << 2 | membrane
                            if ((h.type & ~kHitWalk) > 1) edgeTypes |= 1u << (fk & 3u);
                            uint32_t at = 0;
                            while (at < nkeys && keys[at] != fk) at++;
                            if (at == nkeys) {
                                if (nkeys == (uint32_t)kParitySlots) { st |= kStatusParityOverflow; continue; }
                                keys[nkeys++] = fk;
                            }
                            parity ^= 1u << at;
                        }
                    }
            uint32_t c = 0, f = 0xFFFFu, mt = 0;
            for (; mt < 3 && c == 0; mt++) {
                uint32_t best = 0xFFFFFFFFu;
                for (uint32_t q = 0; q < nkeys; q++)
                    if (((parity >> q) & 1u) && (keys[q] & 3u) == mt) best = min(best, keys[q] >> 2);
                if (best != 0xFFFFFFFFu) {
                    c = (mt == 0) ? 1u : ((mt == 2) ? 3u : 2u);
                    f = best & 0xFFFFu;
                }
            }
            if (edgeTypes & ((1u << mt) - 1u)) continue;  // as above
            resolved = true;
            comp = c;
            fiber = f;
        }
    }
    if (!resolved) st |= kStatusUnresolved;
    S.x[i] = s.x; S.y[i] = s.y; S.z[i] = s.z;
    S.meta[i] = (comp & 0xFFu) | (fiber << 8);
    if (nMoves) atomicAdd(moved, nMoves);
    if (st) atomicOr(status, st);
}

int launch_compartments(const MeshDev& g, const AccelDev& acc, uint64_t entries, const SpinsSorted& S,
                        const float maxabs[3], float startBox, uint64_t seed, uint32_t maxTries, uint32_t maxMoves,
                        uint32_t* status, uint32_t* moved, cudaStream_t st) {
    if (S.N == 0) return kOk;
    // A thread per spin from 100,000 spins on and a quarter of the lists' entries more
    // (long lists keep a warp's lanes busy and a thread's warp waiting for its fullest
    // line), fewer where a line has fewer layers than a warp lanes.  us by a warp / a thread,
    // * the rule's: 2304 triangles, 112 cells per axis (76,000 entries), 60,000 spins
    // 104* / 166, 200,000 262 / 215*, 1M 1200 / 487*; 30,720 triangles (405,000) 100,000
    // 202* / 240, 400,000 701 / 512*; 204,800 triangles (1.76M) 200,000 724* / 991, 1M
    // 3436 / 3068*; at 8 cells per axis 30,000 1223 / 1442*, 200,000 6789 / 2541*.
    const double cells = (double)acc.nf * acc.nf;
    double line = 1e5 + 0.24 * (double)entries * fmin(1.0, 25000.0 / cells);
    if (acc.nf < 24) line *= acc.nf / 24.0;
    if ((double)S.N >= line) {
        const uint32_t grid = (uint32_t)(((uint64_t)S.N + 127) / 128);
        k_compartments_thread<<<grid, 128, 0, st>>>(g, acc, S, maxabs[0], maxabs[1], maxabs[2], startBox,
                                                    (uint32_t)seed, (uint32_t)(seed >> 32), maxTries, maxMoves, status,
                                                    moved);
        DSIM_CUDA_TRY(cudaGetLastError());
        return kOk;
    }
    const uint32_t grid = (uint32_t)(((uint64_t)S.N + 3) / 4);
    k_compartments_warp<<<grid, 128, 0, st>>>(g, acc, S, maxabs[0], maxabs[1], maxabs[2], startBox, (uint32_t)seed,
                                              (uint32_t)(seed >> 32), maxTries, maxMoves, status, moved);
    DSIM_CUDA_TRY(cudaGetLastError());
    return kOk;
}

}  // namespace dsim
