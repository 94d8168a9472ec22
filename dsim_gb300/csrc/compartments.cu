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
// Here one warp follows one spin's line through the fine acceleration grid:
// lane l takes the layers l, l + 32, ... of cells across the line's main axis,
// looks up the cells the line passes there and tests the records of those whose
// slab it may meet.  A crossing is counted only in the cell that contains the
// crossing point, so a triangle listed in several cells counts once.  Crossing
// parity is kept per (fiber, membrane), lane s holding entry s of the list.
// The reference takes its candidates from an R-tree in tree order; when two
// fibers of the same membrane type both enclose a spin (overlapping meshes)
// it keeps the last one in that order, while this kernel keeps the lowest
// fiber index.  For meshes without overlaps the result is the same.
// Tilts and moves draw from Philox keyed by the caller's seed and the spin.
//
// Bound by the latency of the dependent loads (cell, record, triangle): a thread
// per spin walked a hundred layers in turn, its warp as many records as the
// fullest of 32 lines; 100,001 spins on 640,000 triangles took 1.22 ms, now 0.58.
#include "common.cuh"
#include "engine.h"
#include "mesh_common.cuh"

namespace dsim {

static constexpr int kParitySlots = 32;

__device__ __forceinline__ float sgn_ref(float v) { return (v >= 0.0f) ? 1.0f : -1.0f; }

// a lane's walk over its share of the line's cells and their records
struct LineWalk {
    uint32_t ca, cb, cc, lob, hib, loc, hic;  // layer, cell in it and the layer's range
    uint32_t k, end;                          // records of the cell
};

__global__ void __launch_bounds__(128) k_compartments(MeshDev g, AccelDev acc, SpinsSorted S, float mx, float my,
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
            // spinSystem.cpp:1659-1665: a new random position in the start box
            const u32x4 r = philox4x32_10({id, move, 0u, 0xB0C5u}, key0, key1);
            sx = startBox * 2.0f * ((float)(r.x >> 8) * 0x1p-24f - 0.5f);
            sy = startBox * 2.0f * ((float)(r.y >> 8) * 0x1p-24f - 0.5f);
            sz = startBox * 2.0f * ((float)(r.z >> 8) * 0x1p-24f - 0.5f);
            nMoves++;
        }
        for (uint32_t tr = 0; tr <= maxTries && !resolved; tr++) {
            float ex = sx, ey = sy, ez = sz;
            const float ax = fabsf(sx), ay = fabsf(sy), az = fabsf(sz);
            if ((ax > ay) & (ax > az)) ex = (float)((double)sgn_ref(sx) * 1.1 * (double)mx);
            else if (ay > az) ey = (float)((double)sgn_ref(sy) * 1.1 * (double)my);
            else ez = (float)((double)sgn_ref(sz) * 1.1 * (double)mz);
            if (tr > 0) {
                const u32x4 r = philox4x32_10({id, tr, move, 0xC0A5u}, key0, key1);
                ex = (float)((double)ex + (double)((float)(r.x >> 8) * 0x1p-24f) * 0.05);
                ey = (float)((double)ey + (double)((float)(r.y >> 8) * 0x1p-24f) * 0.05);
                ez = (float)((double)ez + (double)((float)(r.z >> 8) * 0x1p-24f) * 0.05);
            }
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

int launch_compartments(const MeshDev& g, const AccelDev& acc, const SpinsSorted& S, const float maxabs[3],
                        float startBox, uint64_t seed, uint32_t maxTries, uint32_t maxMoves, uint32_t* status,
                        uint32_t* moved, cudaStream_t st) {
    if (S.N == 0) return kOk;
    const uint32_t grid = (uint32_t)(((uint64_t)S.N + 3) / 4);
    k_compartments<<<grid, 128, 0, st>>>(g, acc, S, maxabs[0], maxabs[1], maxabs[2], startBox, (uint32_t)seed,
                                         (uint32_t)(seed >> 32), maxTries, maxMoves, status, moved);
    DSIM_CUDA_TRY(cudaGetLastError());
    return kOk;
}

}  // namespace dsim
