// cyl_common.cuh -- the dSim2 membrane rules for one step of one spin, shared
// by the cylinder step kernel (cyl.cu) and the multi-job batch kernels: one
// statement of the rules (cyl_membranes) over three forms of the position --
// FP32 (Cyl32), FP64 (Cyl64) and FP32 offsets from a lattice (CylLocal).
//
// Reference (rfdougherty/dSim): cpuIntegrate dSim2/src/spinKernelCpu.cpp:312-641,
// distToCenterSq :71-82, calcCubePos/calcCubeHash dSim2/src/spinSystem.cpp:413-433.
#pragma once
#include "common.cuh"
#include "engine.h"

namespace dsim {

template <class T>
struct P3 {
    T x, y, z;
};
// a point's grid cell: coordinates and index
struct CylCell {
    uint32_t x, y, z, cube;
};
// d^2 against the squared inner radius (inLt: below, inGt: above) and the
// squared radius of a fiber; touch: the point may lie in the fiber (d^2 <= r^2
// in this form's arithmetic, with a margin where the form rounds positions
// between steps)
struct CylSides {
    bool inLt, inGt, outLt, outGt, touch;
};

// ---- FP32: the reference's arithmetic ---------------------------------------
__device__ __forceinline__ float cyl_dist_sq(float px, float py, float pz, float4 f) {
    if (f.x == 2.0f) return (pz - f.z) * (pz - f.z) + (py - f.y) * (py - f.y);
    else if (f.z == 2.0f) return (px - f.x) * (px - f.x) + (py - f.y) * (py - f.y);
    return (px - f.x) * (px - f.x) + (pz - f.z) * (pz - f.z);
}

// calcCubeHash(calcCubePos(p)): the float3 division of the reference's header
// multiplies by the reciprocal (inv); clamping happens in the hash.  The
// reference's float products (float)(n*n) * cz etc. are exact integers while
// n^3 < 2^24 (its grid has at most 100 cells per axis), so integer arithmetic
// gives the same index.
__device__ __forceinline__ CylCell cyl_cell(uint32_t n, float inv, float px, float py, float pz) {
    const float hi = (float)(n - 1);
    CylCell c;
    c.x = uint_small(fmaxf(fminf(floor_small((px + 1.0f) * inv), hi), 0.0f));
    c.y = uint_small(fmaxf(fminf(floor_small((py + 1.0f) * inv), hi), 0.0f));
    c.z = uint_small(fmaxf(fminf(floor_small((pz + 1.0f) * inv), hi), 0.0f));
    c.cube = n * (n * c.z + c.y) + c.x;
    return c;
}

// The point's fine cell inside its grid cell c (the grid's own cell of the
// point): the fine coordinate, clamped to the grid cell's fineK cells.
__device__ __forceinline__ uint32_t cyl_fine_cell(const CylDev& g, float px, float py, float pz, const CylCell& c) {
    const uint32_t k = g.fineK, nk = g.n * k;
    const float hi = (float)(k - 1);
    const float sx = fminf(fmaxf(floor_small((px + 1.0f) * g.fineInv) - (float)(c.x * k), 0.0f), hi);
    const float sy = fminf(fmaxf(floor_small((py + 1.0f) * g.fineInv) - (float)(c.y * k), 0.0f), hi);
    const float sz = fminf(fmaxf(floor_small((pz + 1.0f) * g.fineInv) - (float)(c.z * k), 0.0f), hi);
    return ((c.z * k + uint_small(sz)) * nk + (c.y * k + uint_small(sy))) * nk + c.x * k + uint_small(sx);
}

struct Cyl32 {
    typedef float T;
    float inR;  // (inner radius proportion)^2
    __device__ __forceinline__ CylSides sides(const P3<float>& p, float4 f) {
        const float cur = cyl_dist_sq(p.x, p.y, p.z, f), A = inR * f.w, B = f.w;
        return {cur < A, cur > A, cur < B, cur > B, !(cur > B)};
    }
    __device__ __forceinline__ CylCell cell(const CylDev& g, const P3<float>& p) const {
        return cyl_cell(g.n, g.inv, p.x, p.y, p.z);
    }
    __device__ __forceinline__ uint32_t fine(const CylDev& g, const P3<float>& p, const CylCell& c) const {
        return cyl_fine_cell(g, p.x, p.y, p.z, c);
    }
};

// ---- FP64 (DSIM_JOB_PRECISE) --------------------------------------------------
// Parameters are the reference's float values (fiber records, r^2, inner radius
// proportion squared, permeability, draws) promoted to double; every
// position-dependent quantity that a result keeps is formed in double in the
// same order.  A decision (a side of a membrane, a grid cell) is taken from FP32
// where its error cannot change it and from the double value otherwise: this
// chip's FP64 pipe runs at 1/64 of the FP32 rate, and a warp's step waited for
// some 11 FP64 operations and 4 conversions in every list entry it tested.
// 13,586 spins, 196 steps: 6.3 -> 3.1 ms alone.
__device__ __forceinline__ double cyl_dist_sq64(double px, double py, double pz, float4 f) {
    const double fx = f.x, fy = f.y, fz = f.z;
    if (f.x == 2.0f) return (pz - fz) * (pz - fz) + (py - fy) * (py - fy);
    else if (f.z == 2.0f) return (px - fx) * (px - fx) + (py - fy) * (py - fy);
    return (px - fx) * (px - fx) + (pz - fz) * (pz - fz);
}

// floor((p + 1) inv), at most hi and at least 0.  The FP32 product t is off by
// less than 5 u (1 + |p|) inv, u = 2^-24 (p, 1 + p, inv and the product are
// rounded once each), so its floor stands unless t lies within twice that of an
// integer.
__device__ __forceinline__ uint32_t cyl_floor64(double p, double inv, uint32_t hi) {
    const float pf = (float)p, vf = (float)inv;
    const float t = (pf + 1.0f) * vf, fl = floor_small(t), m = 6e-7f * (1.0f + fabsf(pf)) * vf;
    if (t - fl > m && t - fl < 1.0f - m) return uint_small(fmaxf(fminf(fl, (float)hi), 0.0f));
    return (uint32_t)fmax(fmin(floor((p + 1.0) * inv), (double)hi), 0.0);
}

struct Cyl64 {
    typedef double T;
    double inR;  // a float's value
    // The FP32 d^2, u = 2^-24 and |p| the largest coordinate: a coordinate e =
    // p - f is off by u (|p| + |e|), so d^2 by u (6 d^2 + 2.83 |p| d) + 2 (u
    // |p|)^2, and the FP32 inR r^2 by u inR r^2.  The band is 4x their sum at d^2
    // = max(inR r^2, r^2) = M, with room for M = 0; farther out d^2 - M grows
    // faster than the error.
    __device__ __forceinline__ CylSides sides(const P3<double>& p, float4 f) {
        const float px = (float)p.x, py = (float)p.y, pz = (float)p.z;
        const float c = cyl_dist_sq(px, py, pz, f), a = (float)inR * f.w, b = f.w;
        const float M = fmaxf(a, b), pm = fmaxf(fabsf(px), fmaxf(fabsf(py), fabsf(pz)));
        const float band = 2.4e-7f * (7.0f * M + 2.83f * pm * sqrtf(M)) + 1e-12f * (pm * pm);
        if (fabsf(c - a) > band && fabsf(c - b) > band) return {c < a, !(c < a), c < b, !(c < b), c < b};
        const double cur = cyl_dist_sq64(p.x, p.y, p.z, f), A = inR * (double)f.w, B = f.w;
        return {cur < A, cur > A, cur < B, cur > B, !(cur > B)};
    }
    __device__ __forceinline__ CylCell cell(const CylDev& g, const P3<double>& p) const {
        CylCell c;
        c.x = cyl_floor64(p.x, g.inv64, g.n - 1);
        c.y = cyl_floor64(p.y, g.inv64, g.n - 1);
        c.z = cyl_floor64(p.z, g.inv64, g.n - 1);
        c.cube = g.n * (g.n * c.z + c.y) + c.x;
        return c;
    }
    // the fine lists are registered in double against cells widened by 1e-5, so
    // every entry able to act at p is in the list of the cell this picks
    __device__ __forceinline__ uint32_t fine(const CylDev& g, const P3<double>& p, const CylCell& c) const {
        const uint32_t k = g.fineK, nk = g.n * k;
        const double inv = (double)g.fineInv;
        const uint32_t fx = min(max(cyl_floor64(p.x, inv, nk - 1), c.x * k), c.x * k + k - 1);
        const uint32_t fy = min(max(cyl_floor64(p.y, inv, nk - 1), c.y * k), c.y * k + k - 1);
        const uint32_t fz = min(max(cyl_floor64(p.z, inv, nk - 1), c.z * k), c.z * k + k - 1);
        return (fz * nk + fy) * nk + fx;
    }
};

// ---- the cell-local FP32 form (DSIM_JOB_LOCAL cylinder jobs) ---------------
// A position is a lattice origin G (a multiple of 1/16, exact in float) plus an
// FP32 offset p.  The distance to a fiber's axis is formed in the local frame,
// ((G - f) + p) per axis, which rounds about 16x finer than the absolute FP32
// coordinates of the reference's step.  Each membrane decision compares d^2
// with inR r^2 and r^2; where the FP32 d^2 lies within its error band of
// either, the decision is taken from the FP64 distance at the exact position
// G + p, as the FP64 form would take it there.  Grid and fine-grid lookups use
// the absolute position rounded to float (the fine lists are registered
// against cells widened by 1e-5).
struct CylOrigin {
    float x, y, z;
};

__device__ __forceinline__ float cyl_dist_sq_local(const CylOrigin& G, float px, float py, float pz, float4 f) {
    if (f.x == 2.0f) {
        const float ez = (G.z - f.z) + pz, ey = (G.y - f.y) + py;
        return ez * ez + ey * ey;
    } else if (f.z == 2.0f) {
        const float ex = (G.x - f.x) + px, ey = (G.y - f.y) + py;
        return ex * ex + ey * ey;
    }
    const float ex = (G.x - f.x) + px, ez = (G.z - f.z) + pz;
    return ex * ex + ez * ez;
}

// d^2 against inR r^2 and r^2.  Error of the FP32 d^2, u = 2^-24: a local
// coordinate e = (G - f) + p is off by at most u (|G - f| + |e|) <=
// u (2|e| + |p|) (two roundings); the squares and the sum add u d^2 each, so
// d^2 is off by at most u (6 d^2 + 2.83 |p| d), and the FP32 threshold inR r^2
// by u inR r^2.  The band is 4x their sum at d^2 = max(inR r^2, r^2) = M; it
// also covers the rounding of the offset when the origin moves.  nexact counts
// the FP64 decisions.
struct CylLocal {
    typedef float T;
    float inR;
    CylOrigin G;
    uint32_t ntests, nexact;
    __device__ __forceinline__ CylSides sides(const P3<float>& p, float4 f) {
        ntests++;
        const float cur = cyl_dist_sq_local(G, p.x, p.y, p.z, f);
        const float A = inR * f.w, B = f.w;
        const float M = fmaxf(A, B);
        const float pm = fmaxf(fabsf(p.x), fmaxf(fabsf(p.y), fabsf(p.z)));
        const float band = 2.4e-7f * (7.0f * M + 2.83f * pm * sqrtf(M));
        if (fabsf(cur - A) > band && fabsf(cur - B) > band)
            return {cur < A, !(cur < A), cur < B, !(cur < B), !(cur > B + band)};
        nexact++;
        const double c = cyl_dist_sq64((double)G.x + (double)p.x, (double)G.y + (double)p.y,
                                       (double)G.z + (double)p.z, f);
        const double A64 = (double)inR * (double)f.w, B64 = (double)f.w;
        return {c < A64, c > A64, c < B64, c > B64, !(cur > B + band)};
    }
    __device__ __forceinline__ CylCell cell(const CylDev& g, const P3<float>& p) const {
        return cyl_cell(g.n, g.inv, G.x + p.x, G.y + p.y, G.z + p.z);
    }
    __device__ __forceinline__ uint32_t fine(const CylDev& g, const P3<float>& p, const CylCell& c) const {
        return cyl_fine_cell(g, G.x + p.x, G.y + p.y, G.z + p.z, c);
    }
};

// ---- the rules ----------------------------------------------------------------
// One list entry (fiber record f, list position j()) of the first pass of a
// spin outside every fiber, tested at the current p.
template <class F, class Pos>
__device__ __forceinline__ void cyl_outside_entry(F& form, float4 f, const uint32_t* list, Pos j,
                                                  const P3<typename F::T>& o, P3<typename F::T>& p,
                                                  typename F::T u, typename F::T perm, uint32_t& imo,
                                                  uint32_t& nearest, uint32_t& nrej, uint32_t& nperm, bool& moved,
                                                  bool& inside, bool& touch) {
    typedef typename F::T T;
    const CylSides s = form.sides(p, f);
    inside |= s.inLt | s.outLt;
    touch |= s.touch;
    if (!s.outGt & s.inGt) {
        if (u >= perm) { p = o; nrej++; moved = true; }
        else { imo = 1; nearest = __ldg(list + j()); nperm++; }
    } else if (s.inLt) {
        if (u < (T)1 - perm) { p = o; nrej++; moved = true; }
        else if (((T)1 - perm < u) & (u < (T)1 - perm * perm)) {
            p = o; nearest = __ldg(list + j()); imo = 1; nrej++;
            moved = true;
        } else { imo = 0; nearest = __ldg(list + j()); nperm++; }
    }
}

// entry j of a grid cell's list: the inline record when the grid has them (the
// index is read only when the spin changes region), else the index and then
// the fiber; false for an index past the fibers
__device__ __forceinline__ bool cyl_entry(const CylDev& g, uint32_t cube, uint32_t j, float4& f, uint32_t& status) {
    const size_t at = (size_t)cube * g.maxFPC + j;
    if (g.cube_fibers) {
        f = __ldg(g.cube_fibers + at);
        return true;
    }
    const uint32_t fi = __ldg(g.cubes + at);
    if (fi >= g.nF) { status |= kStatusBadCell; return false; }
    f = __ldg(g.fibers + fi);
    return true;
}

// Membrane test of the proposed position p (from o) for a spin in region imo
// (0 core, 1 myelin, 2 outside) with nearest fiber `nearest`: a rejected step
// puts p back to o; permeation and the end-position region update imo.
//
// clear (kept by the caller from step to step, false when unknown): no entry of
// o's own grid cell touches o.  A rejected step of such a spin ends at once:
// what the reference still tests is at o, the rest of the list if it is o's
// cell's and the whole second pass, and none of it can act.  (About one step
// in seven is rejected at C1, so nearly every warp used to run these passes.)
// No lane outside leaves before the end: lanes that returned early never met
// the others again, and the long walks over a whole list ran one lane at a time
// (one step of 100,001 spins among 256 cylinders 58 us, and 78 with the returns).
template <class F>
__device__ __forceinline__ void cyl_membranes(const CylDev& g, F& form, const P3<typename F::T>& o,
                                              P3<typename F::T>& p, typename F::T u, typename F::T perm,
                                              uint32_t& imo, uint32_t& nearest, uint32_t& nrej, uint32_t& nperm,
                                              uint32_t& status, bool& clear) {
    typedef typename F::T T;
    if (!(perm < (T)1)) return;
    if (imo < 2) {
        const float4 f = __ldg(g.fibers + nearest);
        const CylSides s = form.sides(p, f);
        if (imo == 0) {
            if (s.inGt & !s.outGt) {
                if (u >= perm) { p = o; nrej++; }
                else { imo = 1; nperm++; }
            } else if (s.outGt) {
                if (u < (T)1 - perm) { p = o; nrej++; }
                else if (((T)1 - perm < u) & (u < (T)1 - perm * perm)) { p = o; imo = 1; nrej++; }
                else { imo = 2; nperm++; }
            }
        } else {
            if (s.outGt) {
                if (u >= perm) { p = o; nrej++; }
                else { imo = 2; nperm++; }
            } else if (s.inLt) {
                if (u >= perm) { p = o; nrej++; }
                else { imo = 0; nperm++; }
            }
        }
        const CylSides e = form.sides(p, f);
        imo = e.outGt ? 2u : (e.inLt ? 0u : 1u);
        clear = false;
        return;
    }
    CylCell c = form.cell(g, p);
    // The second pass below rejects the step once for each fiber of the end
    // position's cell with d^2 < inR r^2 or d^2 < r^2.  While this pass moves
    // nothing, the end position is the one tested here, so `inside` (that test
    // on every entry) decides whether the second pass can change anything; if
    // not, it is skipped.
    bool moved = false, inside = false, touch = false;
    const bool fine = g.fine_start != nullptr && form.inR <= (T)1;
    uint32_t j = 0, cnt = 0;
    if (fine) {
        // While the tested point is p, only the fine cell's entries can act;
        // after the first rejection (p = o) the rest of the list is tested at o.
        const uint32_t fc = form.fine(g, p, c);
        const uint32_t e1 = __ldg(g.fine_start + fc + 1);
        const uint32_t* list = g.cubes + (size_t)c.cube * g.maxFPC;
        uint32_t em = 0;
        for (uint32_t e = __ldg(g.fine_start + fc); e < e1; e++) {
            cyl_outside_entry(form, __ldg(g.fine_rec + e), list, [&] { return __ldg(g.fine_pos + e); }, o, p, u, perm,
                              imo, nearest, nrej, nperm, moved, inside, touch);
            if (moved) { em = e; break; }
        }
        if (!moved) {
            clear = !touch;
        } else {
            const CylCell co = form.cell(g, o);
            if (co.cube != c.cube) {
                j = __ldg(g.fine_pos + em) + 1;
                cnt = __ldg(g.cube_count + c.cube);
            } else if (!clear) {
                const uint32_t jm = __ldg(g.fine_pos + em);
                // the entries after position jm, at o: o's fine cell holds every
                // one that can act there
                const uint32_t fo = form.fine(g, o, co);
                const uint32_t eo1 = __ldg(g.fine_start + fo + 1);
                for (uint32_t e = __ldg(g.fine_start + fo); e < eo1; e++) {
                    const uint32_t jj = __ldg(g.fine_pos + e);
                    if (jj <= jm) continue;
                    cyl_outside_entry(form, __ldg(g.fine_rec + e), list, [&] { return jj; }, o, p, u, perm, imo, nearest,
                                      nrej, nperm, moved, inside, touch);
                }
            }
        }
    } else {
        clear = false;
        cnt = __ldg(g.cube_count + c.cube);
    }
    for (; j < cnt; j++) {
        float4 f;
        if (cyl_entry(g, c.cube, j, f, status))
            cyl_outside_entry(form, f, g.cubes + (size_t)c.cube * g.maxFPC, [&] { return j; }, o, p, u, perm, imo,
                              nearest, nrej, nperm, moved, inside, touch);
    }
    if (imo == 2 && (moved || inside) && !(moved && clear)) {
        c = form.cell(g, p);
        if (fine && moved) {
            // p = o for the whole pass, so o's fine cell stands for the list
            const uint32_t fc = form.fine(g, p, c);
            const uint32_t e1 = __ldg(g.fine_start + fc + 1);
            touch = false;
            for (uint32_t e = __ldg(g.fine_start + fc); e < e1; e++) {
                const CylSides s = form.sides(p, __ldg(g.fine_rec + e));
                touch |= s.touch;
                if (s.inLt | s.outLt) { p = o; nrej++; }
            }
            clear = !touch;
        } else {
            cnt = __ldg(g.cube_count + c.cube);
            for (uint32_t j2 = 0; j2 < cnt; j2++) {
                float4 f;
                if (!cyl_entry(g, c.cube, j2, f, status)) continue;
                const CylSides s = form.sides(p, f);
                if (s.inLt | s.outLt) { p = o; nrej++; }
            }
            clear = false;  // p may have moved
        }
    }
}

// the clamp to the box (the reference's comparisons); a moved point is no
// longer the one the membranes saw
template <class T>
__device__ __forceinline__ void cyl_clamp(P3<T>& p, T lo, T hi, bool& clear) {
    const P3<T> q = p;
    if (p.x > hi) p.x = hi; else if (p.x < lo) p.x = lo;
    if (p.y > hi) p.y = hi; else if (p.y < lo) p.y = lo;
    if (p.z > hi) p.z = hi; else if (p.z < lo) p.z = lo;
    clear = clear & (p.x == q.x) & (p.y == q.y) & (p.z == q.z);
}

}  // namespace dsim
