// accel.cu -- the fine acceleration grid of a mesh, spin sorting by fine
// cell, and the reference-layout transposes of the dSim3 drop-in.
//
// Fine grid: every triangle is listed in every fine cell it touches (a
// separating-axis test in double against the cell widened by kAccelEps), so a
// triangle that the reference's float test reports as hit by a sub-segment is
// always in the lists of the fine cells of the sub-segment's box.  The step
// kernels (flat.cu, batch.cu) collect their hits from these lists and replay
// the reference's grid traversal over them (dSim3/src/spinKernelCpu.cpp:198-395).
//
// Spins are reordered by the Morton code of their fine cell every few steps
// so that the threads of a warp read the same cell records (broadcast loads)
// and the records of a block's cells stay in L1.  Each spin keeps a stable id
// that keys its Philox counter, its replay draws and its counters.
#include "common.cuh"
#include "engine.h"
#include "mesh_common.cuh"

namespace dsim {

// ---- build --------------------------------------------------------------
__device__ __forceinline__ void tri_fine_range(const TriPlane& P, const TriBary& B, float invLf,
                                               uint32_t nf, uint32_t lo[3], uint32_t hi[3]) {
    float p1[3] = {P.p1x, P.p1y, P.p1z};
    float u[3] = {B.ux, B.uy, B.uz};
    float v[3] = {B.vx, B.vy, B.vz};
#pragma unroll
    for (int k = 0; k < 3; k++) {
        float a = p1[k], b = p1[k] + v[k], c = p1[k] + u[k];
        float mn = fminf(a, fminf(b, c)) - kAccelEps;
        float mx = fmaxf(a, fmaxf(b, c)) + kAccelEps;
        lo[k] = fine_coord(mn, invLf, nf);
        hi[k] = fine_coord(mx, invLf, nf);
    }
}

// Separating-axis test of a triangle (corners relative to the box centre)
// against a box of half-extent h: the triangle's plane normal and the nine
// cross products of box axes with triangle edges.  The three box axes are
// already satisfied by the cell range (the triangle's widened bounding box).
// Evaluated in double on float inputs, with the box widened by kAccelEps, so
// every cell the float triangle touches passes.
__device__ __forceinline__ bool tri_box_overlap(const double v[3][3], const double h[3]) {
    const double e0[3] = {v[1][0] - v[0][0], v[1][1] - v[0][1], v[1][2] - v[0][2]};
    const double e1[3] = {v[2][0] - v[1][0], v[2][1] - v[1][1], v[2][2] - v[1][2]};
    const double e2[3] = {v[0][0] - v[2][0], v[0][1] - v[2][1], v[0][2] - v[2][2]};
    const double* E[3] = {e0, e1, e2};
#pragma unroll
    for (int i = 0; i < 3; i++) {      // box axis i
#pragma unroll
        for (int j = 0; j < 3; j++) {  // triangle edge j: axis = unit_i x E[j]
            double a[3] = {0.0, 0.0, 0.0};
            const int i1 = (i + 1) % 3, i2 = (i + 2) % 3;
            a[i1] = -E[j][i2];
            a[i2] = E[j][i1];
            const double p0 = a[0] * v[0][0] + a[1] * v[0][1] + a[2] * v[0][2];
            const double p1 = a[0] * v[1][0] + a[1] * v[1][1] + a[2] * v[1][2];
            const double p2 = a[0] * v[2][0] + a[1] * v[2][1] + a[2] * v[2][2];
            const double r = h[0] * fabs(a[0]) + h[1] * fabs(a[1]) + h[2] * fabs(a[2]);
            const double mn = fmin(p0, fmin(p1, p2)), mx = fmax(p0, fmax(p1, p2));
            if (mn > r || mx < -r) return false;
        }
    }
    const double n[3] = {e0[1] * e1[2] - e0[2] * e1[1], e0[2] * e1[0] - e0[0] * e1[2], e0[0] * e1[1] - e0[1] * e1[0]};
    const double d = n[0] * v[0][0] + n[1] * v[0][1] + n[2] * v[0][2];
    const double r = h[0] * fabs(n[0]) + h[1] * fabs(n[1]) + h[2] * fabs(n[2]);
    return fabs(d) <= r;
}

// The same axes in FP32, deciding only what is clear of rounding: 0 apart, 1
// overlap, 2 too close to call (the FP64 axes decide, so the lists are the
// same).  v: corners relative to the box centre, h: the widened half-extents,
// W the largest of their sizes, u = 2^-24.  A corner is off by u W, an edge
// component by 4 u W, so an edge axis' projections and h . |a| are each
// within 20 u W^2 of the exact ones; a component of the normal is within
// 48 u W^2, its projections within 240 u W^3.  FP64 runs at 1/64 of the FP32
// rate here: with the FP64 axes alone a pass over 640,000 triangles took
// 2.66 ms, with this in front of them 0.47 ms.
__device__ __forceinline__ int tri_box_overlap32(const float v[3][3], const float h[3]) {
    const float e0[3] = {v[1][0] - v[0][0], v[1][1] - v[0][1], v[1][2] - v[0][2]};
    const float e1[3] = {v[2][0] - v[1][0], v[2][1] - v[1][1], v[2][2] - v[1][2]};
    const float e2[3] = {v[0][0] - v[2][0], v[0][1] - v[2][1], v[0][2] - v[2][2]};
    const float* E[3] = {e0, e1, e2};
    float W = fmaxf(h[0], fmaxf(h[1], h[2]));
#pragma unroll
    for (int c = 0; c < 3; c++)
#pragma unroll
        for (int k = 0; k < 3; k++) W = fmaxf(W, fabsf(v[c][k]));
    // also infinite; a NaN is passed over by the maximum, and a triangle with one
    // reports no hit (its normal has one), whatever cells list it
    if (!(W < 4.0f)) return 2;
    const float err2 = 64.0f * 5.9604645e-08f * W * W, err3 = 512.0f * 5.9604645e-08f * W * W * W;
    bool sure = true;
#pragma unroll
    for (int i = 0; i < 3; i++) {
#pragma unroll
        for (int j = 0; j < 3; j++) {
            const int i1 = (i + 1) % 3, i2 = (i + 2) % 3;
            const float a1 = -E[j][i2], a2 = E[j][i1];
            const float p0 = a1 * v[0][i1] + a2 * v[0][i2], p1 = a1 * v[1][i1] + a2 * v[1][i2],
                        p2 = a1 * v[2][i1] + a2 * v[2][i2];
            const float r = h[i1] * fabsf(a1) + h[i2] * fabsf(a2);
            const float gap = fmaxf(fminf(p0, fminf(p1, p2)), -fmaxf(p0, fmaxf(p1, p2))) - r;  // > 0: apart
            if (gap > err2) return 0;
            sure &= gap < -err2;
        }
    }
    const float n[3] = {e0[1] * e1[2] - e0[2] * e1[1], e0[2] * e1[0] - e0[0] * e1[2], e0[0] * e1[1] - e0[1] * e1[0]};
    const float d = n[0] * v[0][0] + n[1] * v[0][1] + n[2] * v[0][2];
    const float gap = fabsf(d) - (h[0] * fabsf(n[0]) + h[1] * fabsf(n[1]) + h[2] * fabsf(n[2]));
    if (gap > err3) return 0;
    sure &= gap < -err3;
    return sure ? 1 : 2;
}

// box of fine cell index k on one axis, widened by kAccelEps; the outermost
// cells reach to infinity because coordinates beyond the box clamp into them
__device__ __forceinline__ void cell_span(uint32_t k, uint32_t nf, double& lo, double& hi) {
    const double Lf = 2.0 / (double)nf;
    lo = (k == 0) ? -1.0e6 : -1.0 + (double)k * Lf - (double)kAccelEps;
    hi = (k == nf - 1) ? 1.0e6 : -1.0 + (double)(k + 1) * Lf + (double)kAccelEps;
}

// The corners of a triangle relative to the middle of cell k on one axis, in
// float (the middle to 1e-15, against 1e-9 that tri_box_overlap32 allows for)
struct CellAxis {
    float v[3];
};
__device__ __forceinline__ CellAxis cell_axis(uint32_t k, double Lf, float c0, float c1, float c2) {
    const double ctr = -1.0 + ((double)k + 0.5) * Lf;
    CellAxis a;
    a.v[0] = (float)((double)c0 - ctr);
    a.v[1] = (float)((double)c1 - ctr);
    a.v[2] = (float)((double)c2 - ctr);
    return a;
}

// Pass 1 counts, pass 2 fills.  touched: per triangle of up to kMaskCells cells
// in its range, the ones pass 1 found it in by their order, so that pass 2 tests
// none again; a larger triangle's are tested in both.  The FP64 parts of a test
// are formed once per cell of each axis.  640,000 triangles: count 0.45 -> 0.30
// ms, fill 0.50 -> 0.09 ms.
template <bool FILL>
__global__ void k_accel_cells(uint32_t nT, const TriPlane* __restrict__ plane,
                              const TriBary* __restrict__ bary, uint32_t nf, float invLf,
                              uint32_t* counter, const uint32_t* __restrict__ start, AccelRec* rec,
                              uint32_t* tri, AccelRecWide* recw, AccelRecFull* recf, uint64_t* touched) {
    uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nT) return;
    TriPlane P = plane[t];
    TriBary B = bary[t];
    uint32_t lo[3], hi[3];
    tri_fine_range(P, B, invLf, nf, lo, hi);
    // corners as the intersection test sees the triangle: p1, p1 + v, p1 + u
    const float c0[3] = {P.p1x, P.p1y, P.p1z};
    const float c1[3] = {P.p1x + B.vx, P.p1y + B.vy, P.p1z + B.vz};
    const float c2[3] = {P.p1x + B.ux, P.p1y + B.uy, P.p1z + B.uz};
    const uint64_t cells = (uint64_t)(hi[0] - lo[0] + 1) * (hi[1] - lo[1] + 1) * (hi[2] - lo[2] + 1);
    const bool many = cells > 1, masked = cells <= kMaskCells, test = many && !(FILL && masked);
    uint64_t mask = FILL && masked ? touched[t] : 0ull, bit = 1ull;
    // the outermost cells are open: left to the FP64 axes
    const double Lf = 2.0 / (double)nf;
    const float hf = (float)(0.5 * Lf + (double)kAccelEps);
    const float h32[3] = {hf, hf, hf};
    CellAxis ax = {}, ay = {}, az;
    for (uint32_t x = lo[0]; x <= hi[0]; x++) {
        if (test) ax = cell_axis(x, Lf, c0[0], c1[0], c2[0]);
        for (uint32_t y = lo[1]; y <= hi[1]; y++) {
            if (test) ay = cell_axis(y, Lf, c0[1], c1[1], c2[1]);
            for (uint32_t z = lo[2]; z <= hi[2]; z++, bit <<= 1) {
                if (test) {
                    az = cell_axis(z, Lf, c0[2], c1[2], c2[2]);
                    const float v32[3][3] = {{ax.v[0], ay.v[0], az.v[0]},
                                             {ax.v[1], ay.v[1], az.v[1]},
                                             {ax.v[2], ay.v[2], az.v[2]}};
                    const bool open = min(x, min(y, z)) == 0 || max(x, max(y, z)) == nf - 1;
                    const int clear = open ? 2 : tri_box_overlap32(v32, h32);
                    if (clear == 0) continue;
                    if (clear == 2) {
                        const uint32_t at[3] = {x, y, z};
                        double v[3][3], h[3];
                        for (int k = 0; k < 3; k++) {
                            double bl, bh;
                            cell_span(at[k], nf, bl, bh);
                            const double ctr = 0.5 * (bl + bh);
                            h[k] = 0.5 * (bh - bl);
                            v[0][k] = (double)c0[k] - ctr;
                            v[1][k] = (double)c1[k] - ctr;
                            v[2][k] = (double)c2[k] - ctr;
                        }
                        if (!tri_box_overlap(v, h)) continue;
                    }
                } else if (FILL && masked && !(mask & bit)) {
                    continue;
                }
                if (!FILL) mask |= bit;
                uint32_t key = morton3(x, y, z);
                uint32_t slot = atomicAdd(counter + key, 1u);
                if (FILL) {
                    const float4 q = make_float4(P.nx, P.ny, P.nz, P.nx * P.p1x + P.ny * P.p1y + P.nz * P.p1z);
                    if (recf) {
                        AccelRecFull r;
                        r.a = make_float4(P.nx, P.ny, P.nz, P.vv);
                        r.b = make_float4(P.p1x, P.p1y, P.p1z, __uint_as_float(t));
                        r.c = make_float4(B.ux, B.uy, B.uz, B.vx);
                        r.d = make_float4(B.vy, B.vz, B.uv, B.uu);
                        recf[start[key] + slot] = r;
                    } else if (recw) {
                        AccelRecWide r;
                        r.q = q;
                        r.pt = make_float4(P.p1x, P.p1y, P.p1z, __uint_as_float(t));
                        recw[start[key] + slot] = r;
                    } else {
                        AccelRec r;
                        r.q = q;
                        rec[start[key] + slot] = r;
                        tri[start[key] + slot] = t;
                    }
                }
            }
        }
    }
    if (!FILL && masked) touched[t] = mask;
}

int launch_accel_cells(bool fill, uint32_t nT, const TriPlane* plane, const TriBary* bary,
                       uint32_t nf, uint32_t* counter, const uint32_t* start, AccelRec* rec,
                       uint32_t* tri, AccelRecWide* recw, uint64_t* touched, cudaStream_t st, AccelRecFull* recf) {
    if (nT == 0) return kOk;
    float invLf = (float)nf / 2.0f;
    if (fill)
        k_accel_cells<true><<<(nT + 127) / 128, 128, 0, st>>>(nT, plane, bary, nf, invLf, counter, start, rec, tri, recw, recf, touched);
    else
        k_accel_cells<false><<<(nT + 127) / 128, 128, 0, st>>>(nT, plane, bary, nf, invLf, counter, start, rec, tri, recw, recf, touched);
    DSIM_CUDA_TRY(cudaGetLastError());
    return kOk;
}

// ---- cell slabs -----------------------------------------------------------
// How far a point the float triangle test reports on triangle (u, v) may lie
// off the triangle, normalised units.  kSlabEps covers the rounding of
// positions, crossing points and of N . x on both sides (a few 1e-7 each); the
// rest is the rounding of the Gram system behind the barycentric coordinates,
// about 40 ulps of the triangle's size over sin^2 of its angle at p1 (64
// taken).  Infinite, so that its cells cull nothing, for a triangle whose
// Gram system is nearly singular.
static constexpr float kSlabEps = 2.5e-5f;
__device__ __forceinline__ float slab_margin(const TriBary& B, float vv) {
    const float uu = fabsf(B.uu);
    const float s2 = 1.0f - (B.uv / uu) * (B.uv / vv);
    if (!(s2 > 1e-5f) || !(uu > 0.0f) || !(vv > 0.0f)) return 1e30f;
    return kSlabEps + 64.0f * 5.9604645e-08f * sqrtf(fmaxf(uu, vv)) / s2;
}

// Marks (by the sign of vv) the triangles whose hits need the reference's walk
// over its cells: those that enter the inside of some reference cell (shrunk
// by kRegularEps) that does not list them, that lie in more than four cells,
// or whose float test may report a point farther off (slab_margin).  Any other
// triangle is listed by the cell of a hit point that keeps 2 kRegularEps from
// the cell's faces (flat_only_hit).  walkAll: every one (a plug-in host whose cell
// edge is not 2 / n: the walk then visits other cells than those that hold a
// point).  The reference's overlap test is decided by
// rounding where a triangle ends on a face, as the rings of a tessellated tube
// often do, so touching a face alone says nothing.  The sign of uu tells a test
// to look vv up: it is flagged, or not v . v to the last bit (tri_vv).
__global__ void k_tri_regular(uint32_t nT, uint32_t n, bool walkAll, const uint4* __restrict__ cells,
                              TriBary* bary, TriPlane* plane) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nT) return;
    const float eps = kRegularEps;
    const TriPlane P = plane[t];
    const TriBary B = bary[t];
    const uint4 c = cells[t];
    const float vv = fabsf(P.vv), inv = 0.5f * (float)n, L = 2.0f / (float)n;
    const float c0[3] = {P.p1x, P.p1y, P.p1z};
    const float c1[3] = {P.p1x + B.vx, P.p1y + B.vy, P.p1z + B.vz};
    const float c2[3] = {P.p1x + B.ux, P.p1y + B.uy, P.p1z + B.uz};
    uint32_t lo[3], hi[3];
    float mn[3], mx[3];
    bool regular = !walkAll && c.x != kCellMany && slab_margin(B, vv) <= eps;
    for (int k = 0; k < 3; k++) {
        mn[k] = fminf(c0[k], fminf(c1[k], c2[k]));
        mx[k] = fmaxf(c0[k], fmaxf(c1[k], c2[k]));
        regular = regular && mn[k] > -2.0f && mx[k] < 2.0f;
    }
    for (int k = 0; regular && k < 3; k++) {
        lo[k] = fine_coord(mn[k], inv, n);
        hi[k] = fine_coord(mx[k], inv, n);
        regular = hi[k] - lo[k] < 6u;  // four cells at most are listed
    }
    for (uint32_t x = regular ? lo[0] : 1u; regular && x <= hi[0]; x++)
        for (uint32_t y = lo[1]; regular && y <= hi[1]; y++)
            for (uint32_t z = lo[2]; regular && z <= hi[2]; z++) {
                const uint32_t at = x | (y << 10) | (z << 20);
                if (c.x == at || c.y == at || c.z == at || c.w == at) continue;
                const uint32_t q[3] = {x, y, z};
                float v[3][3], h[3];
                bool apart = false;
                for (int k = 0; k < 3; k++) {
                    // the outermost cells are open: to the triangle's own extent
                    float bl = -1.0f + (float)q[k] * L + eps, bh = -1.0f + (float)(q[k] + 1) * L - eps;
                    if (q[k] == 0) bl = fminf(bl, mn[k]);
                    if (q[k] == n - 1) bh = fmaxf(bh, mx[k]);
                    const float ctr = 0.5f * (bl + bh);
                    h[k] = 0.5f * (bh - bl);
                    v[0][k] = c0[k] - ctr; v[1][k] = c1[k] - ctr; v[2][k] = c2[k] - ctr;
                    apart = apart || mn[k] > bh || mx[k] < bl;
                }
                regular = apart || tri_box_overlap32(v, h) == 0;
            }
    plane[t].vv = regular ? vv : -vv;
    if (!regular || vv != B.vx * B.vx + B.vy * B.vy + B.vz * B.vz) bary[t].uu = -fabsf(B.uu);
}

int launch_tri_regular(uint32_t nT, uint32_t n, bool walkAll, const uint4* cells, TriBary* bary, TriPlane* plane,
                       cudaStream_t st) {
    if (nT == 0) return kOk;
    k_tri_regular<<<(nT + 127) / 128, 128, 0, st>>>(nT, n, walkAll, cells, bary, plane);
    DSIM_CUDA_TRY(cudaGetLastError());
    return kOk;
}

// One thread per cell, in the table's order (x fastest).  N is the sum of the
// records' normals, each turned to the first one's side, scaled to its largest
// component 127 and rounded; lo and hi are the range of N . x over the
// records' corners, widened by each triangle's margin times |N|.
__global__ void __launch_bounds__(128) k_accel_slabs(uint32_t nf, const TriPlane* __restrict__ plane,
                                                     const TriBary* __restrict__ bary,
                                                     const uint32_t* __restrict__ start,
                                                     const uint32_t* __restrict__ tri,
                                                     const AccelRecWide* __restrict__ recw,
                                                     const AccelRecFull* __restrict__ recf, AccelCell* cell) {
    const uint32_t x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y, z = blockIdx.z;
    if (x >= nf) return;
    const uint32_t key = morton3(x, y, z);
    const uint32_t b0 = start[key], b1 = start[key + 1];
    AccelCell r;
    r.first = b0; r.slab = 0u; r.lo = -3.0e38f; r.hi = 3.0e38f;
    if (b1 > b0) {
        float sx = 0.0f, sy = 0.0f, sz = 0.0f, rx = 0.0f, ry = 0.0f, rz = 0.0f;
        for (uint32_t k = b0; k < b1; k++) {
            const uint32_t t = recf ? __float_as_uint(recf[k].b.w) : (recw ? __float_as_uint(recw[k].pt.w) : tri[k]);
            const float nx = plane[t].nx, ny = plane[t].ny, nz = plane[t].nz;
            if (k == b0) { rx = nx; ry = ny; rz = nz; }
            const float s = nx * rx + ny * ry + nz * rz < 0.0f ? -1.0f : 1.0f;
            sx += s * nx; sy += s * ny; sz += s * nz;
        }
        const float big = fmaxf(fabsf(sx), fmaxf(fabsf(sy), fabsf(sz)));
        float Nx = 0.0f, Ny = 0.0f, Nz = 0.0f;
        if (big > 0.0f && big < 1e30f && sx == sx && sy == sy && sz == sz) {
            Nx = rintf(sx / big * 127.0f); Ny = rintf(sy / big * 127.0f); Nz = rintf(sz / big * 127.0f);
        }
        const float len = sqrtf(Nx * Nx + Ny * Ny + Nz * Nz);
        float lo = 3.0e38f, hi = -3.0e38f;
        for (uint32_t k = b0; k < b1; k++) {
            const uint32_t t = recf ? __float_as_uint(recf[k].b.w) : (recw ? __float_as_uint(recw[k].pt.w) : tri[k]);
            const TriPlane P = plane[t];
            const TriBary B = bary[t];
            const float a = Nx * P.p1x + Ny * P.p1y + Nz * P.p1z;
            const float u = Nx * B.ux + Ny * B.uy + Nz * B.uz, v = Nx * B.vx + Ny * B.vy + Nz * B.vz;
            const float m = slab_margin(B, fabsf(P.vv)) * len * fmaxf(1.0f, fmaxf(fabsf(P.p1x), fmaxf(fabsf(P.p1y), fabsf(P.p1z))));
            const float l = a + fminf(0.0f, fminf(u, v)) - m, h = a + fmaxf(0.0f, fmaxf(u, v)) + m;
            lo = fminf(lo, l); hi = fmaxf(hi, h);
            if (!(h - l < 1e29f) || !(a + u + v == a + u + v)) { lo = -3.0e38f; hi = 3.0e38f; }
        }
        if (len > 0.0f && lo > -1e29f && hi < 1e29f) { r.lo = lo; r.hi = hi; }
        r.slab = (min(b1 - b0, 255u) << 24) | ((uint32_t)(int)Nx & 0xFFu) | (((uint32_t)(int)Ny & 0xFFu) << 8) |
                 (((uint32_t)(int)Nz & 0xFFu) << 16);
    }
    cell[((size_t)z * nf + y) * nf + x] = r;
}

int launch_accel_slabs(uint32_t nf, const TriPlane* plane, const TriBary* bary, const uint32_t* start,
                       const uint32_t* tri, const AccelRecWide* recw, const AccelRecFull* recf, AccelCell* cell,
                       cudaStream_t st) {
    k_accel_slabs<<<dim3((nf + 127) / 128, nf, nf), 128, 0, st>>>(nf, plane, bary, start, tri, recw, recf, cell);
    DSIM_CUDA_TRY(cudaGetLastError());
    return kOk;
}

// ---- spin sorting (counting sort on a coarse Morton key) -----------------
__global__ void k_sort_keys(SpinsSorted S, uint32_t nb, float invLb, uint32_t* keys, uint32_t* hist) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= S.N) return;
    uint32_t key = morton3(fine_coord(S.x[i], invLb, nb), fine_coord(S.y[i], invLb, nb),
                           fine_coord(S.z[i], invLb, nb));
    keys[i] = key;
    atomicAdd(hist + key, 1u);
}

__global__ void k_sort_scatter(SpinsSorted S, SpinsSorted D, const uint32_t* __restrict__ keys,
                               const uint32_t* __restrict__ start, uint32_t* cursor) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= S.N) return;
    uint32_t key = keys[i];
    uint32_t j = start[key] + atomicAdd(cursor + key, 1u);
    D.x[j] = S.x[i]; D.y[j] = S.y[i]; D.z[j] = S.z[i];
    D.mag[j] = S.mag[i]; D.phase[j] = S.phase[i];
    D.meta[j] = S.meta[i]; D.id[j] = S.id[i];
}

uint32_t sort_grid(uint32_t N, uint32_t nf) {
    uint32_t nb = 8;
    while (nb < nf && (uint64_t)nb * nb * nb < 2ull * N) nb++;
    return nb < nf ? nb : nf;
}

int launch_sort_spins(const SpinsSorted& S, const SpinsSorted& D, uint32_t nb, uint32_t* keys,
                      uint32_t* hist, uint32_t* start, uint32_t* scratch, cudaStream_t st) {
    if (S.N == 0) return kOk;
    uint32_t nkeys = morton3(nb - 1, nb - 1, nb - 1) + 1;
    DSIM_CUDA_TRY(cudaMemsetAsync(hist, 0, (size_t)nkeys * 4, st));
    float invLb = (float)nb / 2.0f;
    k_sort_keys<<<(S.N + 255) / 256, 256, 0, st>>>(S, nb, invLb, keys, hist);
    int rc = launch_scan_exclusive(hist, start, nkeys, scratch, st);
    if (rc) return rc;
    DSIM_CUDA_TRY(cudaMemsetAsync(hist, 0, (size_t)nkeys * 4, st));
    k_sort_scatter<<<(S.N + 255) / 256, 256, 0, st>>>(S, D, keys, start, hist);
    DSIM_CUDA_TRY(cudaGetLastError());
    return kOk;
}

}  // namespace dsim

namespace dsim {
// slot order back to spin order: D[id[i]] = S[i]
__global__ void k_unpermute(SpinsSorted S, SpinsSorted D) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= S.N) return;
    uint32_t j = S.id[i];
    if (j >= S.N) return;
    D.x[j] = S.x[i]; D.y[j] = S.y[i]; D.z[j] = S.z[i];
    D.mag[j] = S.mag[i]; D.phase[j] = S.phase[i]; D.meta[j] = S.meta[i]; D.id[j] = j;
}

int launch_unpermute(const SpinsSorted& S, const SpinsSorted& D, cudaStream_t st) {
    if (S.N == 0) return kOk;
    k_unpermute<<<(S.N + 255) / 256, 256, 0, st>>>(S, D);
    DSIM_CUDA_TRY(cudaGetLastError());
    return kOk;
}
}  // namespace dsim

namespace dsim {
// the reference's AoS arrays (float3 positions, 12-byte spinData) -> SoA
// work buffers in spin order (id = index)
__global__ void k_aos_to_soa(const float* __restrict__ pos, const unsigned char* __restrict__ spin,
                             SpinsSorted D) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= D.N) return;
    D.x[i] = pos[3 * i]; D.y[i] = pos[3 * i + 1]; D.z[i] = pos[3 * i + 2];
    const unsigned char* rec = spin + 12 * (size_t)i;
    D.mag[i] = *reinterpret_cast<const float*>(rec);
    D.phase[i] = *reinterpret_cast<const float*>(rec + 4);
    D.meta[i] = (uint32_t)rec[8] | ((uint32_t)(*reinterpret_cast<const uint16_t*>(rec + 10)) << 8);
    D.id[i] = i;
}

// SoA work buffers (any slot order) -> the reference's AoS arrays by id; with
// spinKeys, each spin's key is advanced for the next call
__global__ void k_soa_to_aos(SpinsSorted S, float* pos, unsigned char* spin, uint32_t* spinKeys,
                             uint32_t iterations) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= S.N) return;
    uint32_t j = S.id[i];
    if (j >= S.N) return;
    pos[3 * j] = S.x[i]; pos[3 * j + 1] = S.y[i]; pos[3 * j + 2] = S.z[i];
    unsigned char* rec = spin + 12 * (size_t)j;
    *reinterpret_cast<float*>(rec) = S.mag[i];
    *reinterpret_cast<float*>(rec + 4) = S.phase[i];
    rec[8] = (unsigned char)(S.meta[i] & 0xFFu);
    *reinterpret_cast<uint16_t*>(rec + 10) = (uint16_t)(S.meta[i] >> 8);
    if (spinKeys) {
        uint32_t k0 = spinKeys[2 * j], k1 = spinKeys[2 * j + 1];
        u32x4 nk = philox4x32_10({j, iterations, 0xFFFFFFFFu, 0x5EEDu}, k0, k1);
        spinKeys[2 * j] = nk.x; spinKeys[2 * j + 1] = nk.y;
    }
}

int launch_aos_to_soa(const float* pos, const void* spin, const SpinsSorted& D, cudaStream_t st) {
    if (D.N == 0) return kOk;
    k_aos_to_soa<<<(D.N + 255) / 256, 256, 0, st>>>(pos, (const unsigned char*)spin, D);
    DSIM_CUDA_TRY(cudaGetLastError());
    return kOk;
}

int launch_soa_to_aos(const SpinsSorted& S, float* pos, void* spin, uint32_t* spinKeys,
                      uint32_t iterations, cudaStream_t st) {
    if (S.N == 0) return kOk;
    k_soa_to_aos<<<(S.N + 255) / 256, 256, 0, st>>>(S, pos, (unsigned char*)spin, spinKeys, iterations);
    DSIM_CUDA_TRY(cudaGetLastError());
    return kOk;
}
}  // namespace dsim

namespace dsim {
// The host's arrays as they come (StageArrays, one buffer on the device) <->
// the work buffers.  Interleaving, widening and the reordering by id were host
// loops over every spin and six copies either way; a null array is left out.
__global__ void k_stage_load(StageArrays A, SpinsSorted D) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= D.N) return;
    if (A.pos) { D.x[i] = A.pos[3 * i]; D.y[i] = A.pos[3 * i + 1]; D.z[i] = A.pos[3 * i + 2]; }
    if (A.mag) D.mag[i] = A.mag[i];
    if (A.phase) D.phase[i] = A.phase[i];
    if (A.comp || A.fiber16)
        D.meta[i] = (A.comp ? (uint32_t)A.comp[i] : 0u) | ((A.fiber16 ? (uint32_t)A.fiber16[i] : 0xFFFFu) << 8);
    D.id[i] = i;
}
__global__ void k_stage_store(SpinsSorted S, StageArrays A) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= S.N) return;
    const uint32_t j = S.id[i];
    if (j >= S.N) return;
    if (A.pos) { A.pos[3 * j] = S.x[i]; A.pos[3 * j + 1] = S.y[i]; A.pos[3 * j + 2] = S.z[i]; }
    if (A.mag) A.mag[j] = S.mag[i];
    if (A.phase) A.phase[j] = S.phase[i];
    if (A.comp) A.comp[j] = (uint8_t)(S.meta[i] & 0xFFu);
    if (A.fiber16) A.fiber16[j] = (uint16_t)(S.meta[i] >> 8);
}
// cylinder spins: word 2 of a seed record is imo + 1 (set: 2 when not given; get:
// a record of 0 reads as outside), word 3 the nearest fiber
__global__ void k_stage_load_cyl(StageArrays A, CylSpinsDev D) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= D.N) return;
    D.pos[i] = make_float4(A.pos[3 * i], A.pos[3 * i + 1], A.pos[3 * i + 2], A.phase ? A.phase[i] : 0.0f);
    reinterpret_cast<uint4*>(D.seed4)[i] =
        make_uint4(0u, 0u, (A.imo ? A.imo[i] : 2u) + 1u, A.nearest ? A.nearest[i] : 0xFFFFFFFFu);
    D.mag[i] = A.mag ? A.mag[i] : 1.0f;
}
__global__ void k_stage_store_cyl(CylSpinsDev S, StageArrays A) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= S.N) return;
    const float4 p = S.pos[i];
    const uint4 w = reinterpret_cast<const uint4*>(S.seed4)[i];
    if (A.pos) { A.pos[3 * i] = p.x; A.pos[3 * i + 1] = p.y; A.pos[3 * i + 2] = p.z; }
    if (A.mag) A.mag[i] = S.mag[i];
    if (A.phase) A.phase[i] = p.w;
    if (A.imo) A.imo[i] = w.z ? w.z - 1u : 2u;
    if (A.nearest) A.nearest[i] = w.w;
}

int launch_stage_load(const StageArrays& A, const SpinsSorted& D, cudaStream_t st) {
    if (D.N == 0) return kOk;
    k_stage_load<<<(D.N + 255) / 256, 256, 0, st>>>(A, D);
    DSIM_CUDA_TRY(cudaGetLastError());
    return kOk;
}
int launch_stage_store(const SpinsSorted& S, const StageArrays& A, cudaStream_t st) {
    if (S.N == 0) return kOk;
    k_stage_store<<<(S.N + 255) / 256, 256, 0, st>>>(S, A);
    DSIM_CUDA_TRY(cudaGetLastError());
    return kOk;
}
int launch_stage_load_cyl(const StageArrays& A, const CylSpinsDev& D, cudaStream_t st) {
    if (D.N == 0) return kOk;
    k_stage_load_cyl<<<(D.N + 255) / 256, 256, 0, st>>>(A, D);
    DSIM_CUDA_TRY(cudaGetLastError());
    return kOk;
}
int launch_stage_store_cyl(const CylSpinsDev& S, const StageArrays& A, cudaStream_t st) {
    if (S.N == 0) return kOk;
    k_stage_store_cyl<<<(S.N + 255) / 256, 256, 0, st>>>(S, A);
    DSIM_CUDA_TRY(cudaGetLastError());
    return kOk;
}
}  // namespace dsim
