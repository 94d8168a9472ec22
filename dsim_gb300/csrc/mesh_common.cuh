// mesh_common.cuh -- device helpers shared by the mesh step kernels (flat.cu,
// batch.cu) and the compartment search: fine-grid coordinates and Morton
// keys, the exact triangle test on a fine-grid record, membership in a
// reference-grid cell, and the reference grid scan used as the exact fallback.
#pragma once
#include "common.cuh"
#include "engine.h"

namespace dsim {

// the fine-grid coordinate of p: floor((p + 1) / Lf) clamped to [0, nf - 1]
// (floor_small / uint_small: the values of floorf and the conversion, on the
// FP32 pipe)
__device__ __forceinline__ uint32_t fine_coord(float p, float invLf, uint32_t nf) {
    float f = floor_small((p + 1.0f) * invLf);
    f = fminf(fmaxf(f, 0.0f), (float)(nf - 1));
    return uint_small(f);
}

__host__ __device__ __forceinline__ uint32_t spread3(uint32_t v) {
    // 10 bits -> every third bit
    v &= 0x3FFu;
    v = (v | (v << 16)) & 0x030000FFu;
    v = (v | (v << 8)) & 0x0300F00Fu;
    v = (v | (v << 4)) & 0x030C30C3u;
    v = (v | (v << 2)) & 0x09249249u;
    return v;
}
__host__ __device__ __forceinline__ uint32_t morton3(uint32_t x, uint32_t y, uint32_t z) {
    return spread3(x) | (spread3(y) << 1) | (spread3(z) << 2);
}

// ---- the step ------------------------------------------------------------
struct FastHit {
    uint32_t t;
    float x, y, z, d2;
    float r;  // the point's fraction of the sub-segment
    uint32_t type;
};
// Hit type flag: the reference's walk over its cells decides whether (and when)
// it meets this triangle.  Without it every reference cell that the triangle
// enters by more than kRegularEps lists it (k_tri_regular; the sign of its vv
// carries the flag), so a sub-segment's only hit is the reference's when it
// lies clear of the cell's faces.
static constexpr float kRegularEps = 3e-5f;
static constexpr uint32_t kHitWalk = 0x200u;
__device__ __forceinline__ uint32_t hit_walk(float vv) { return __float_as_uint(vv) >> 31 << 9; }

// reference-grid membership of triangle t in cell c: binary search of the
// ascending list
__device__ __forceinline__ bool in_ref_cell(const MeshDev& g, uint32_t c, uint32_t t) {
    uint32_t lo = __ldg(g.cell_start + c), hi = __ldg(g.cell_start + c + 1);
    while (lo < hi) {
        uint32_t mid = (lo + hi) >> 1;
        uint32_t v = __ldg(g.cell_tri + mid);
        if (v == t) return true;
        if (v < t) lo = mid + 1; else hi = mid;
    }
    return false;
}

__device__ __forceinline__ uint32_t ref_coord(float p, float L, uint32_t n) {
    float f = floorf((p + 1.0f) / L);
    float hi = (float)(n - 1);
    float mn = (hi < f) ? hi : f;
    float mx = (0.0f < mn) ? mn : 0.0f;
    return (uint32_t)mx;
}

// ---- which of several hits the reference takes ------------------------------
// cubeCollDetect's loops (dSim3/src/spinKernelCpu.cpp:198-337) walk the
// reference cells from the start's to the end's, x outermost and z innermost,
// and stop at the first whose list holds a hit.  A cell's place in that walk is
// (ax ny + ay) nz + az, ax, ay, az its distances from the start's cell, so the
// reference's hit is the one of lowest (place of its triangle's first cell,
// distance, triangle index), found without walking the cells.
static constexpr uint32_t kNoPlace = 0xFFFFFFFFu;
struct RefWalk {
    uint32_t sx, sy, sz;  // the start's cell
    int ix, iy, iz;       // +1, or -1 where the walk descends
    uint32_t nx, ny, nz;  // cells on each axis
};
__device__ __forceinline__ RefWalk ref_walk(uint32_t sx, uint32_t sy, uint32_t sz, uint32_t tx, uint32_t ty,
                                            uint32_t tz) {
    RefWalk w;
    w.sx = sx; w.sy = sy; w.sz = sz;
    w.ix = tx < sx ? -1 : 1; w.iy = ty < sy ? -1 : 1; w.iz = tz < sz ? -1 : 1;
    w.nx = (uint32_t)(w.ix * (int)(tx - sx)) + 1u;
    w.ny = (uint32_t)(w.iy * (int)(ty - sy)) + 1u;
    w.nz = (uint32_t)(w.iz * (int)(tz - sz)) + 1u;
    return w;
}
// does p keep 2 kRegularEps from the faces of its reference cell?
__device__ __forceinline__ bool clear_of_faces(float p, float inv, float margin) {
    const float e = (p + 1.0f) * inv;
    const float f = e - floor_small(e);
    return (f > margin) & (f < 1.0f - margin);
}
// the place of packed cell c (pack_cell), kNoPlace when the walk misses it
__device__ __forceinline__ uint32_t cell_place(const RefWalk& w, uint32_t c) {
    const uint32_t ax = (uint32_t)(w.ix * (int)((c & 1023u) - w.sx));
    const uint32_t ay = (uint32_t)(w.iy * (int)(((c >> 10) & 1023u) - w.sy));
    const uint32_t az = (uint32_t)(w.iz * (int)((c >> 20) - w.sz));  // an unused entry's z is 4095
    return ((ax < w.nx) & (ay < w.ny) & (az < w.nz)) ? (ax * w.ny + ay) * w.nz + az : kNoPlace;
}
// a triangle of more than four cells: walk the cells, searching their lists
static __device__ __noinline__ uint32_t search_place(const MeshDev& g, RefWalk w, uint32_t t) {
    for (uint32_t ax = 0; ax < w.nx; ax++)
        for (uint32_t ay = 0; ay < w.ny; ay++)
            for (uint32_t az = 0; az < w.nz; az++) {
                const uint32_t x = w.sx + (uint32_t)w.ix * ax, y = w.sy + (uint32_t)w.iy * ay,
                               z = w.sz + (uint32_t)w.iz * az;
                if (in_ref_cell(g, g.n * g.n * z + g.n * y + x, t)) return (ax * w.ny + ay) * w.nz + az;
            }
    return kNoPlace;
}
// the place of the first of triangle t's cells (its record `c`, loaded ahead)
__device__ __forceinline__ uint32_t first_place(const MeshDev& g, const RefWalk& w, uint4 c, uint32_t t) {
    if (c.x == kCellMany) return search_place(g, w, t);
    return min(min(cell_place(w, c.x), cell_place(w, c.y)), min(cell_place(w, c.z), cell_place(w, c.w)));
}

// full test of one accel record against the sub-segment (same float
// expressions as triCollDetect); returns true and fills h on a hit
// a = {n, p1.x}, b = {p1.y, p1.z, vv, t}, u4 = {u, v.x}, v4 = {v.y, v.z, uv, uu}
__device__ __forceinline__ bool test_rec_uv(float4 a, float4 b, float4 u4, float4 v4, float ox, float oy,
                                            float oz, float dx, float dy, float dz, FastHit& h) {
    float num = a.x * (a.w - ox) + a.y * (b.x - oy) + a.z * (b.y - oz);
    float den = a.x * dx + a.y * dy + a.z * dz;
    if (!(fabsf(num) <= fabsf(den)) || num == 0.0f ||
        ((__float_as_uint(num) ^ __float_as_uint(den)) & 0x80000000u))
        return false;
    float r = num / den;
    if (!((0.0f < r) & (r < 1.0f))) return false;
    uint32_t t = __float_as_uint(b.w);
    float wx = ox + r * dx - a.w;
    float wy = oy + r * dy - b.x;
    float wz = oz + r * dz - b.y;
    float wu = wx * u4.x + wy * u4.y + wz * u4.z;
    float wv = wx * u4.w + wy * v4.x + wz * v4.y;
    float uv = v4.z, uu = fabsf(v4.w), vv = fabsf(b.z);
    float s = (uv * wv - vv * wu) / (uv * uv - uu * vv);
    float tt = (uv * wu - uu * wv) / (uv * uv - uu * vv);
    if (!((s >= 0.0f) & (tt >= 0.0f) & (s + tt <= 1.0f))) return false;
    h.t = t;
    h.r = r;
    h.x = ox + dx * r; h.y = oy + dy * r; h.z = oz + dz * r;
    h.d2 = (ox - h.x) * (ox - h.x) + (oy - h.y) * (oy - h.y) + (oz - h.z) * (oz - h.z);
    uint32_t type = 1;
    if ((s == 0.0f) | (tt == 0.0f) | (s + tt == 1.0f)) {
        type = 2;
        if (((s == 0.0f) & (tt == 0.0f)) | ((s == 0.0f) & (tt == 1.0f)) | ((s == 1.0f) & (tt == 0.0f)))
            type = 3;
    }
    h.type = type | hit_walk(b.z);
    return true;
}

// the same, reading u, v, uv, uu from the triangle's records
__device__ __forceinline__ bool test_rec(const MeshDev& g, float4 a, float4 b, float ox, float oy,
                                         float oz, float dx, float dy, float dz, FastHit& h) {
    float num = a.x * (a.w - ox) + a.y * (b.x - oy) + a.z * (b.y - oz);
    float den = a.x * dx + a.y * dy + a.z * dz;
    if (!(fabsf(num) <= fabsf(den)) || num == 0.0f ||
        ((__float_as_uint(num) ^ __float_as_uint(den)) & 0x80000000u))
        return false;
    const float4* bb = reinterpret_cast<const float4*>(g.bary + __float_as_uint(b.w));
    return test_rec_uv(a, b, __ldg(bb), __ldg(bb + 1), ox, oy, oz, dx, dy, dz, h);
}

// a 64-byte record already in registers (no dependent load)
__device__ __forceinline__ bool test_full(const AccelRecFull& r, uint32_t excl, float ox, float oy, float oz,
                                          float dx, float dy, float dz, FastHit& h) {
    if (__float_as_uint(r.b.w) == excl) return false;
    return test_rec_uv(make_float4(r.a.x, r.a.y, r.a.z, r.b.x), make_float4(r.b.y, r.b.z, r.a.w, r.b.w), r.c, r.d,
                       ox, oy, oz, dx, dy, dz, h);
}

__device__ __forceinline__ AccelRecFull load_full(const AccelRecFull* p) {
    const float4* q = reinterpret_cast<const float4*>(p);
    AccelRecFull r;
    r.a = __ldg(q); r.b = __ldg(q + 1); r.c = __ldg(q + 2); r.d = __ldg(q + 3);
    return r;
}


// Conservative plane test on a fine-grid record q = {n, n.p1}: with den the
// exact denominator of triCollDetect and na = n.p1 - n.o, the exact numerator
// differs from na by at most ~2.5e-6 for points in the box (a few float
// roundings of terms of size <= 3.5), so a margin of 1e-5 keeps every record
// whose exact test can pass (0 < num/den < 1).
static constexpr float kPlaneMargin = 1e-5f;
__device__ __forceinline__ bool plane_may_cross(float4 q, float ox, float oy, float oz, float dx,
                                                float dy, float dz) {
    // fused sums: a bound, tighter than the separate roundings the margin allows for
    const float den = __fmaf_rn(q.x, dx, __fmaf_rn(q.y, dy, q.z * dz));
    const float na = __fmaf_rn(-q.x, ox, __fmaf_rn(-q.y, oy, __fmaf_rn(-q.z, oz, q.w)));
    return (den > 0.0f) ? ((na > -kPlaneMargin) & (na < den + kPlaneMargin))
                        : ((den < 0.0f) & (na < kPlaneMargin) & (na > den - kPlaneMargin));
}

// The records of fine cell (x, y, z) that the sub-segment o -> o + d can hit:
// first record b0 and count cnt, 0 when both ends lie on the same outer side
// of the cell's slab (the sub-segment then passes every triangle of the cell
// by more than the exact test's rounding, so none can report a hit).  A bound
// and no result of the reference's, so its sums may be fused.  About half of
// the records of the cells a step touches are skipped this way (14.5 -> 7.0
// per spin-step among 100 beaded tubes, 25.3 -> 16.2 where each carries
// myelin).
__device__ __forceinline__ void cell_records(const AccelDev& acc, uint32_t x, uint32_t y, uint32_t z, float ox,
                                             float oy, float oz, float dx, float dy, float dz, uint32_t& b0,
                                             uint32_t& cnt) {
    const uint4 c = __ldg(reinterpret_cast<const uint4*>(acc.cell + ((size_t)z * acc.nf + y) * acc.nf + x));
    b0 = c.x;
    cnt = c.y >> 24;
    const float nx = (float)(int)(signed char)(c.y & 0xFFu), ny = (float)(int)(signed char)((c.y >> 8) & 0xFFu),
                nz = (float)(int)(signed char)((c.y >> 16) & 0xFFu);
    const float so = __fmaf_rn(nx, ox, __fmaf_rn(ny, oy, nz * oz));
    const float sp = so + __fmaf_rn(nx, dx, __fmaf_rn(ny, dy, nz * dz));
    const float lo = __uint_as_float(c.z), hi = __uint_as_float(c.w);
    if ((fmaxf(so, sp) < lo) | (fminf(so, sp) > hi)) cnt = 0;
    else if (cnt == 255u) cnt = __ldg(acc.start + morton3(x, y, z) + 1) - b0;
}

// exact test against triangle t from its per-triangle records
__device__ __forceinline__ bool test_tri(const MeshDev& g, uint32_t t, float ox, float oy, float oz,
                                         float dx, float dy, float dz, FastHit& h) {
    const float4* pp = reinterpret_cast<const float4*>(g.plane + t);
    const float4 a = __ldg(pp), c = __ldg(pp + 1);
    return test_rec(g, a, make_float4(c.x, c.y, c.z, __uint_as_float(t)), ox, oy, oz, dx, dy, dz, h);
}

// vv of triangle t with its flag (hit_walk): v . v, and from the triangle's
// plane record only where the sign of uu says that it is flagged or given
// otherwise (k_tri_regular): a sector a triangle less to fetch
__device__ __forceinline__ float tri_vv(const MeshDev& g, uint32_t t, float4 u4, float4 v4) {
    if (__float_as_uint(v4.w) >> 31) return __ldg(&g.plane[t].vv);
    return u4.w * u4.w + v4.x * v4.x + v4.y * v4.y;
}

// exact test with the plane data from a 32-byte record (p1, t) and the rest
// (u, v, uv, uu) from the triangle's records, loaded only past the plane
__device__ __forceinline__ bool test_split(const MeshDev& g, float4 q, float4 pt, float ox, float oy,
                                           float oz, float dx, float dy, float dz, FastHit& h) {
    float num = q.x * (pt.x - ox) + q.y * (pt.y - oy) + q.z * (pt.z - oz);
    float den = q.x * dx + q.y * dy + q.z * dz;
    if (!(fabsf(num) <= fabsf(den)) || num == 0.0f ||
        ((__float_as_uint(num) ^ __float_as_uint(den)) & 0x80000000u))
        return false;
    float r = num / den;
    if (!((0.0f < r) & (r < 1.0f))) return false;
    const uint32_t t = __float_as_uint(pt.w);
    const float4* bb = reinterpret_cast<const float4*>(g.bary + t);
    const float4 u4 = __ldg(bb), v4 = __ldg(bb + 1);
    return test_rec_uv(make_float4(q.x, q.y, q.z, pt.x), make_float4(pt.y, pt.z, tri_vv(g, t, u4, v4), pt.w), u4, v4,
                       ox, oy, oz, dx, dy, dz, h);
}

// a 16-byte record k (plane in the record, triangle index beside it)
__device__ __forceinline__ bool test_narrow(const MeshDev& g, const AccelDev& acc, uint32_t k, uint32_t excl,
                                            float ox, float oy, float oz, float dx, float dy, float dz, FastHit& h) {
    const float4 q = __ldg(&acc.rec[k].q);
    if (!plane_may_cross(q, ox, oy, oz, dx, dy, dz)) return false;
    const uint32_t t = __ldg(acc.tri + k);
    if (t == excl) return false;
    return test_tri(g, t, ox, oy, oz, dx, dy, dz, h);
}

// one fine-grid entry k against a sub-segment (any record layout)
__device__ __forceinline__ bool test_entry(const MeshDev& g, const AccelDev& acc, uint32_t k,
                                           uint32_t excl, float ox, float oy, float oz, float dx,
                                           float dy, float dz, FastHit& h) {
    if (acc.wide == 2) return test_full(load_full(acc.recf + k), excl, ox, oy, oz, dx, dy, dz, h);
    if (acc.wide) {
        const float4 q = __ldg(&acc.recw[k].q);
        if (!plane_may_cross(q, ox, oy, oz, dx, dy, dz)) return false;
        const float4 pt = __ldg(&acc.recw[k].pt);
        if (__float_as_uint(pt.w) == excl) return false;
        return test_split(g, q, pt, ox, oy, oz, dx, dy, dz, h);
    }
    return test_narrow(g, acc, k, excl, ox, oy, oz, dx, dy, dz, h);
}

// cubeCollDetect over the reference grid (dSim3/src/spinKernelCpu.cpp:311-337)
static __device__ __noinline__ void ref_scan(const MeshDev& g, float ox, float oy, float oz, float px, float py,
                                             float pz, uint32_t excluded, FastHit& best, bool& found) {
    const uint32_t n = g.n;
    const float L = g.L;
    float dx = px - ox, dy = py - oy, dz = pz - oz;
    uint32_t sx = ref_coord(ox, L, n), sy = ref_coord(oy, L, n), sz = ref_coord(oz, L, n);
    uint32_t tx = ref_coord(px, L, n), ty = ref_coord(py, L, n), tz = ref_coord(pz, L, n);
    uint32_t ix = (uint32_t)((int)(tx > sx) - (int)(tx < sx));
    uint32_t iy = (uint32_t)((int)(ty > sy) - (int)(ty < sy));
    uint32_t iz = (uint32_t)((int)(tz > sz) - (int)(tz < sz));
    found = false;
    uint32_t cx = sx;
    do {
        uint32_t cy = sy;
        do {
            uint32_t cz = sz;
            do {
                uint32_t c = n * n * cz + n * cy + cx;
                uint32_t b0 = __ldg(g.cell_start + c), b1 = __ldg(g.cell_start + c + 1);
                float bd2 = 400000000.0f;
                for (uint32_t k = b0; k < b1; k++) {
                    uint32_t t = __ldg(g.cell_tri + k);
                    if (t == excluded) continue;
                    const float4* pp = reinterpret_cast<const float4*>(g.plane + t);
                    float4 ra = __ldg(pp), rc = __ldg(pp + 1);
                    float4 rb = make_float4(rc.x, rc.y, rc.z, __uint_as_float(t));
                    FastHit h;
                    if (!test_rec(g, ra, rb, ox, oy, oz, dx, dy, dz, h)) continue;
                    if (h.d2 < bd2) { bd2 = h.d2; best = h; best.type &= ~kHitWalk; found = true; }
                }
                cz += iz;
            } while ((cz != tz + iz) && !found);
            cy += iy;
        } while ((cy != ty + iy) && !found);
        cx += ix;
    } while ((cx != tx + ix) && !found);
}

}  // namespace dsim
