// batch.cu -- many simulation jobs advanced by one step launch per chunk
// (include/dsim_batch.h).
//
// Spins of all jobs live in one packed SoA array; job j owns the slot range
// [slot0_j, slot0_j + pad_j) with pad_j = nSpins rounded up to 32, so every
// warp belongs to one job and reads that job's substrate and parameters once.
// Padding slots carry id 0xFFFFFFFF and do no work.  Every chunk the spins
// are re-sorted by (job, Morton cell of a per-job sort grid; for cylinder jobs
// region and scattered id) -- the job ranges are preserved because job j's keys follow job j-1's -- and one step
// kernel advances every running job by up to `chunk` steps.  The chunk loop
// (sort, step, step-counter advance) is captured in a CUDA graph.
//
// Step rules: mesh jobs run the flattened collision round of flat_round.cuh
// (dSim3/src/spinKernelCpu.cpp:198-499), cylinder jobs the dSim2 rules of
// cyl_common.cuh (dSim2/src/spinKernelCpu.cpp:312-641).  Draws are Philox with
// key = job seed and counter = (spin index in the job, job step, 0), the same
// as dsim_mesh_run / dsim_cyl_run with that seed.  Instead of the reference's
// float phase (dSim3/src/spinKernelCpu.cpp:490) each spin accumulates the
// gradient moment M = sum w(t) pos(t) with Kahan compensation; the phase of any
// gradient sharing the waveform is phaseConstant * (g . M), in FP64 at readout.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#pragma GCC visibility push(default)
#include "../../include/dsim_batch.h"
#pragma GCC visibility pop
#include "common.cuh"
#include "cyl_common.cuh"
#include "engine.h"
#include "flat_round.cuh"
#include "local_round.cuh"
#include "prec_round.cuh"

namespace dsim {

enum SubKind : uint32_t { kSubMesh = 0, kSubCyl = 1 };
struct SubDev {
    uint32_t kind;
    MeshDev g;
    AccelDev acc;
    CylDev c;
};

struct JobDev {
    uint32_t sub, steps, start;  // substrate, total steps, global step of the job's step 0
    uint32_t sortBase, sortBits;  // first sort key, Morton bits per axis of the sort grid
    float sd[4], T2[4];
    float perm, dt, clampHi, clampLo;
    uint32_t reflType, maxSub;
    float inR;                    // cylinders: (inner radius proportion)^2
    const float* wave;            // w[steps]
    uint32_t key0, key1;
    uint32_t flags;               // DSIM_JOB_PRECISE or DSIM_JOB_LOCAL
    float spinR;                  // spin radius (the precision form clamps to +-(1 - spinR) in FP64)
    uint32_t sortRegion;          // cylinders: spins outside every fiber sort after those inside, each kind by id
};

static_assert(sizeof(JobDev) % 4 == 0 && sizeof(SubDev) % 4 == 0, "records are copied by 32-bit words");

// packed spin state; meta = compartment | fiber << 8 (cylinders: imo | nearest << 8)
static constexpr int kBF = 10;  // float fields: x y z mx my mz cx cy cz mag
static constexpr int kBU = 3;   // uint fields: meta job id
static constexpr int kBD = 4;   // double fields of precision-form jobs: x y z mag (null until the first one)
struct BatchSpins {
    float* f[kBF];
    uint32_t* u[kBU];
    double* d[kBD];
    uint32_t N;
};
enum { F_X, F_Y, F_Z, F_MX, F_MY, F_MZ, F_CX, F_CY, F_CZ, F_MAG };
enum { U_META, U_JOB, U_ID };
enum { D_X, D_Y, D_Z, D_MAG };

__device__ __forceinline__ void kahan_add(float& s, float& c, float v) {
    float y = v - c;
    float t = s + y;
    c = (t - s) - y;
    s = t;
}

// The warps of one kind of step kernel: first slot, number of slots (of one
// job) and the stride between them of each, at most `per` slots (spins_per_warp
// over the kind's spins).  A launch covers the kind's unfinished jobs only,
// whatever else the batch holds.  Mesh slots are dealt out (kDealWarps).
struct StepWarps {
    const uint2* warp;  // first slot; number | stride << 8
    uint32_t count, per;
};
struct WarpSlots {
    uint32_t first, n, stride;
    __device__ __forceinline__ uint32_t slot(uint32_t at) const { return first + min(at, n - 1u) * stride; }
};
__device__ __forceinline__ WarpSlots warp_slots(const StepWarps& W, uint32_t w) {
    const uint2 q = __ldg(W.warp + w);
    return {q.x, q.y & 0xFFu, q.y >> 8};
}

// Draws for a warp whose lanes repeat its `per` spins (a power of two; lane l
// holds spin l mod per): every 32 / per steps all lanes draw at once, lane l for
// its spin's step number l / per of the coming ones, and a step takes its draw
// by shuffles.  live: the lanes with a spin, by a ballot of the whole warp (inside
// the branch of those lanes nothing makes them run together, and __activemask
// would name whichever did).
struct ThinDraws {
    Draw drawn;
    __device__ __forceinline__ Draw step(uint32_t it, uint32_t per, uint32_t lane, uint32_t live, uint32_t id,
                                         uint32_t step0, uint32_t k0, uint32_t k1) {
        const uint32_t lg = 31u - __clz(per), k = it & ((32u >> lg) - 1u);
        if (k == 0) drawn = philox_draw(id, (uint64_t)(step0 + it + (lane >> lg)), 0u, k0, k1);
        if (per == 32) return drawn;
        const uint32_t from = (k << lg) + (lane & (per - 1u));
        Draw d;
        d.nx = __shfl_sync(live, drawn.nx, from);
        d.ny = __shfl_sync(live, drawn.ny, from);
        d.nz = __shfl_sync(live, drawn.nz, from);
        d.u = __shfl_sync(live, drawn.u, from);
        return d;
    }
};

// The plain form has one instantiation per fine-grid record layout (LAYOUT 1:
// 32-byte, 2: 64-byte records), each advancing only the mesh jobs whose
// substrate uses it, and one for cylinder jobs (LAYOUT 3), so no kernel
// carries the registers of a path it does not run.  Precision-form and
// cell-local jobs run in k_batch_step64 and k_batch_step_local.  THREADS:
// block size (64, 128 or 256); MINB counts 128-thread blocks per SM, so every
// block shape of one occupancy has the same register budget per thread.
// Mesh lanes keep what a round does not read in shared memory (LaneState), and
// 32-byte records past the plane test are finished 32 at a time (FlatQueue):
// 52,000 mesh and 52,000 cylinder spins in six jobs 11.5 -> 10.6 ms for 800
// steps.
template <int MINB, int LAYOUT, int THREADS = kFlatThreads>
__global__ void __launch_bounds__(THREADS, MINB * kFlatThreads / THREADS)
k_batch_step(const SubDev* __restrict__ subs, const JobDev* __restrict__ jobs, BatchSpins S, StepWarps W,
             const uint32_t* __restrict__ stepNow, uint32_t chunk, uint32_t* status,
             unsigned long long* jobCounts) {
    constexpr int MESH = LAYOUT == 3 ? 1 : LAYOUT;  // the record path of the mesh instantiations
    __shared__ FlatWarp wh[LAYOUT == 3 ? 1 : THREADS / 32];
    __shared__ LaneState wc[LAYOUT == 3 ? 1 : THREADS / 32];
    __shared__ FlatQueue wq[LAYOUT == 1 ? THREADS / 32 : 1];
    // gradient moments and their compensation live in shared memory (touched
    // once per step), which keeps the collision loop's registers free
    __shared__ float mom[6][THREADS];
    const uint32_t FULL = 0xFFFFFFFFu;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t tx = threadIdx.x;
    FlatWarp& H = wh[LAYOUT == 3 ? 0u : (threadIdx.x >> 5)];  // the cylinder path uses no table
    const uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (w >= W.count) return;  // whole warp
    // mesh: the lanes past the warp's spins help with the records; cylinders:
    // they repeat the spins (ThinDraws)
    const WarpSlots mine = warp_slots(W, w);
    const uint32_t at = LAYOUT == 3 ? lane & (W.per - 1u) : lane;
    const uint32_t i = mine.slot(at);
    const uint32_t jb = S.u[U_JOB][mine.first];
    // the warp's job and substrate records, copied to shared memory once and
    // read from there (kept out of the collision loop's registers)
    __shared__ JobDev jobS[THREADS / 32];
    __shared__ SubDev subS[THREADS / 32];
    const uint32_t wi = threadIdx.x >> 5;
    {
        const uint32_t* src = reinterpret_cast<const uint32_t*>(jobs + jb);
        uint32_t* dst = reinterpret_cast<uint32_t*>(jobS + wi);
        for (uint32_t k = lane; k < sizeof(JobDev) / 4; k += 32) dst[k] = __ldg(src + k);
        __syncwarp();
        const uint32_t* s2 = reinterpret_cast<const uint32_t*>(subs + jobS[wi].sub);
        uint32_t* d2 = reinterpret_cast<uint32_t*>(subS + wi);
        for (uint32_t k = lane; k < sizeof(SubDev) / 4; k += 32) d2[k] = __ldg(s2 + k);
        __syncwarp();
    }
    const JobDev& J = jobS[wi];
    const uint32_t now = *stepNow;
    const uint32_t start = J.start, steps = J.steps;
    if (now < start || now - start >= steps) return;  // not started or finished (warp-uniform)
    const uint32_t ls0 = now - start;
    const uint32_t nsteps = min(chunk, steps - ls0);
    const uint32_t id = S.u[U_ID][i];
    const bool valid = id != 0xFFFFFFFFu && at < mine.n;
    float x = S.f[F_X][i], y = S.f[F_Y][i], z = S.f[F_Z][i];
    mom[0][tx] = S.f[F_MX][i]; mom[1][tx] = S.f[F_MY][i]; mom[2][tx] = S.f[F_MZ][i];
    mom[3][tx] = S.f[F_CX][i]; mom[4][tx] = S.f[F_CY][i]; mom[5][tx] = S.f[F_CZ][i];
    float mag = S.f[F_MAG][i];
    const uint32_t meta = S.u[U_META][i];
    uint32_t comp = meta & 0xFFu, fiber = meta >> 8;
    uint32_t nrefl = 0, nperm = 0, st = 0;
    const SubDev& sub = subS[wi];
    const uint32_t live = LAYOUT == 3 ? __ballot_sync(FULL, valid) : 0u;  // ThinDraws
    if (LAYOUT != 3) {
        const MeshDev& g = sub.g;
        const AccelDev& acc = sub.acc;
        LaneState& C = wc[LAYOUT == 3 ? 0u : wi];
        float &cmag = C.mag[lane], &umax = C.umax[lane], &umin = C.umin[lane], &u = C.u[lane];
        uint32_t &ccomp = C.comp[lane], &cfiber = C.fiber[lane], &crefl = C.nrefl[lane], &cperm = C.nperm[lane],
                 &status = C.status[lane], &it = C.it[lane], &sub_n = C.sub[lane];
        cmag = mag; ccomp = comp; cfiber = fiber;
        umax = u = 1.0f; umin = 0.0f;
        crefl = cperm = status = it = sub_n = 0;
        bool active = valid && nsteps > 0;
        bool fresh = active;
        // the position is o at the top of a step, the start of its current sub-segment within one
        float ox = x, oy = y, oz = z, px = x, py = y, pz = z;
        uint32_t excluded = 0xFFFFFFFFu;
        while (__any_sync(FULL, active)) {
            if (fresh) {
                const Draw d = philox_draw(id, (uint64_t)(ls0 + it), 0u, J.key0, J.key1);
                u = d.u;
                const float sd = J.sd[ccomp & 3u];
                px = ox + d.nx * sd; py = oy + d.ny * sd; pz = oz + d.nz * sd;
                excluded = 0xFFFFFFFFu;
                umax = 1.0f; umin = 0.0f;
                sub_n = 0;
                fresh = false;
            }
            const bool open = active;
            bool found;
            FastHit best;
            flat_round_mode<MESH>(H, g, acc, lane, open, ox, oy, oz, px, py, pz, excluded, found, best,
                                  LAYOUT == 1 ? &wq[LAYOUT == 1 ? wi : 0u] : nullptr);
            if (open) {
                bool finish = !found;
                if (found) {
                    apply_hit(g, best, u, J.perm, J.reflType, umax, umin, ox, oy, oz, px, py, pz, ccomp, cfiber,
                              excluded, crefl, cperm);
                    if (++sub_n >= J.maxSub) {
                        status |= kStatusSubsegCap;
                        px = ox; py = oy; pz = oz;
                        finish = true;
                    }
                }
                if (finish) {
                    float ex = px, ey = py, ez = pz;
                    if (ex > J.clampHi) ex = J.clampHi; else if (ex < J.clampLo) ex = J.clampLo;
                    if (ey > J.clampHi) ey = J.clampHi; else if (ey < J.clampLo) ey = J.clampLo;
                    if (ez > J.clampHi) ez = J.clampHi; else if (ez < J.clampLo) ez = J.clampLo;
                    ox = ex; oy = ey; oz = ez;
                    const float T2 = J.T2[ccomp & 3u];
                    if (T2 > 0.0f) cmag += -cmag / T2 * J.dt;
                    const float w = __ldg(J.wave + ls0 + it);
                    kahan_add(mom[0][tx], mom[3][tx], w * ox);
                    kahan_add(mom[1][tx], mom[4][tx], w * oy);
                    kahan_add(mom[2][tx], mom[5][tx], w * oz);
                    if (++it >= nsteps) active = false;
                    else fresh = true;
                }
            }
            __syncwarp();
        }
        x = ox; y = oy; z = oz;
        mag = cmag; comp = ccomp; fiber = cfiber; nrefl = crefl; nperm = cperm; st = status;
    } else if (valid) {
        ThinDraws draws;
        const uint32_t k0 = J.key0, k1 = J.key1;
        const float* __restrict__ wave = J.wave;
        const CylDev& g = sub.c;
        const float perm = J.perm;
        uint32_t imo = comp, nearest = fiber;
        Cyl32 form = {J.inR};
        bool clear = false;
        if (imo < 2 && nearest >= g.nF) imo = 2;
        for (uint32_t it = 0; it < nsteps; it++) {
            const Draw d = draws.step(it, W.per, lane, live, id, ls0, k0, k1);
            const float sdv = J.sd[imo];
            const P3<float> o = {x, y, z};
            P3<float> p = {x + d.nx * sdv, y + d.ny * sdv, z + d.nz * sdv};
            cyl_membranes(g, form, o, p, d.u, perm, imo, nearest, nrefl, nperm, st, clear);
            cyl_clamp(p, J.clampLo, J.clampHi, clear);
            x = p.x; y = p.y; z = p.z;
            const float T2 = J.T2[imo];
            if (T2 > 0.0f) mag += -mag / T2 * J.dt;
            const float w = __ldg(wave + ls0 + it);
            kahan_add(mom[0][tx], mom[3][tx], w * x);
            kahan_add(mom[1][tx], mom[4][tx], w * y);
            kahan_add(mom[2][tx], mom[5][tx], w * z);
        }
        comp = imo;
        fiber = nearest & 0xFFFFFFu;
    }
    const bool own = valid && lane == at;
    if (own) {
        S.f[F_X][i] = x; S.f[F_Y][i] = y; S.f[F_Z][i] = z;
        S.f[F_MX][i] = mom[0][tx]; S.f[F_MY][i] = mom[1][tx]; S.f[F_MZ][i] = mom[2][tx];
        S.f[F_CX][i] = mom[3][tx]; S.f[F_CY][i] = mom[4][tx]; S.f[F_CZ][i] = mom[5][tx];
        S.f[F_MAG][i] = mag;
        S.u[U_META][i] = (comp & 0xFFu) | (fiber << 8);
    }
    // per-job counters {reflections, permeations}: one atomic per warp
    unsigned long long r = own ? nrefl : 0u, p = own ? nperm : 0u;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        r += __shfl_down_sync(FULL, r, o);
        p += __shfl_down_sync(FULL, p, o);
    }
    if (lane == 0) {
        if (r) atomicAdd(jobCounts + 4 * jb, r);
        if (p) atomicAdd(jobCounts + 4 * jb + 1, p);
    }
    if (st) atomicOr(status, st);
}

// Cell-local FP32 mesh jobs (DSIM_JOB_LOCAL): the plain step with positions
// as FP32 offsets from a lattice origin (local_round.cuh), FP64 re-tests of
// near-degenerate intersections, Kahan moments.  Between chunks the position
// is kept in the double fields as origin + offset; the float fields get its
// rounded value (sort keys, float readers).
// 4 blocks per SM: the round's two queues and FP64 re-test take 128 registers
// (ms of runs of 200 steps at 4 / 5 / 6: 65,536 mesh spins 6.9 / 6.9 / 7.9,
// 196,608 20.5 / 20.4 / 23.1).
template <int LAYOUT>
__global__ void __launch_bounds__(kFlatThreads, 4)
k_batch_step_local(const SubDev* __restrict__ subs, const JobDev* __restrict__ jobs, BatchSpins S, StepWarps W,
                   const uint32_t* __restrict__ stepNow, uint32_t chunk, uint32_t* status,
                   unsigned long long* jobCounts) {
    __shared__ HitWarp wh[kFlatWarps];
    __shared__ LaneState wc[kFlatWarps];
    __shared__ LocalWarp wl[kFlatWarps];
    __shared__ float mom[6][kFlatThreads];
    __shared__ JobDev jobS[kFlatWarps];
    __shared__ SubDev subS[kFlatWarps];
    const uint32_t FULL = 0xFFFFFFFFu;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t tx = threadIdx.x;
    const uint32_t wi = threadIdx.x >> 5;
    HitWarp& H = wh[wi];
    LocalWarp& Lw = wl[wi];
    const uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (w >= W.count) return;  // whole warp
    const WarpSlots mine = warp_slots(W, w);
    const uint32_t i = mine.slot(lane);
    const uint32_t jb = S.u[U_JOB][mine.first];
    {
        const uint32_t* src = reinterpret_cast<const uint32_t*>(jobs + jb);
        uint32_t* dst = reinterpret_cast<uint32_t*>(jobS + wi);
        for (uint32_t k = lane; k < sizeof(JobDev) / 4; k += 32) dst[k] = __ldg(src + k);
        __syncwarp();
        const uint32_t* s2 = reinterpret_cast<const uint32_t*>(subs + jobS[wi].sub);
        uint32_t* d2 = reinterpret_cast<uint32_t*>(subS + wi);
        for (uint32_t k = lane; k < sizeof(SubDev) / 4; k += 32) d2[k] = __ldg(s2 + k);
        __syncwarp();
    }
    const JobDev& J = jobS[wi];
    const uint32_t now = *stepNow;
    const uint32_t start = J.start, steps = J.steps;
    if (now < start || now - start >= steps) return;
    const uint32_t ls0 = now - start;
    const uint32_t nsteps = min(chunk, steps - ls0);
    const uint32_t id = S.u[U_ID][i];
    const bool valid = id != 0xFFFFFFFFu && lane < mine.n;
    // position = lattice origin (multiple of 1/16) + FP32 offset in [0, 1/16)
    float &gx = Lw.gx[lane], &gy = Lw.gy[lane], &gz = Lw.gz[lane];  // local_round keeps it there too
    gx = gy = gz = 0.0f;
    float ox = 0.0f, oy = 0.0f, oz = 0.0f;
    LaneState& C = wc[wi];
    float &mag = C.mag[lane], &umax = C.umax[lane], &umin = C.umin[lane], &u = C.u[lane];
    uint32_t &comp = C.comp[lane], &fiber = C.fiber[lane], &nrefl = C.nrefl[lane], &nperm = C.nperm[lane],
             &st = C.status[lane], &it = C.it[lane], &sub_n = C.sub[lane];
    mag = umin = 0.0f;
    umax = u = 1.0f;
    comp = fiber = nrefl = nperm = st = it = sub_n = 0;
    mom[0][tx] = 0.0f; mom[1][tx] = 0.0f; mom[2][tx] = 0.0f;
    mom[3][tx] = 0.0f; mom[4][tx] = 0.0f; mom[5][tx] = 0.0f;
    if (valid) {
        const double X = S.d[D_X][i], Y = S.d[D_Y][i], Z = S.d[D_Z][i];
        const double Gx = floor(X * 16.0) * 0.0625, Gy = floor(Y * 16.0) * 0.0625, Gz = floor(Z * 16.0) * 0.0625;
        gx = (float)Gx; gy = (float)Gy; gz = (float)Gz;
        ox = (float)(X - Gx); oy = (float)(Y - Gy); oz = (float)(Z - Gz);
        mag = S.f[F_MAG][i];
        mom[0][tx] = S.f[F_MX][i]; mom[1][tx] = S.f[F_MY][i]; mom[2][tx] = S.f[F_MZ][i];
        mom[3][tx] = S.f[F_CX][i]; mom[4][tx] = S.f[F_CY][i]; mom[5][tx] = S.f[F_CZ][i];
        const uint32_t meta = S.u[U_META][i];
        comp = meta & 0xFFu; fiber = meta >> 8;
    }
    const MeshDev& g = subS[wi].g;
    const AccelDev& acc = subS[wi].acc;
    uint32_t excluded = 0xFFFFFFFFu;
    PrecCount pc;
    bool active = valid && nsteps > 0;
    bool fresh = active;
    // the position is o at the top of a step, the start of its current sub-segment within one
    float px = ox, py = oy, pz = oz;
    while (__any_sync(FULL, active)) {
        if (fresh) {
            const Draw d = philox_draw(id, (uint64_t)(ls0 + it), 0u, J.key0, J.key1);
            u = d.u;
            const float sd = J.sd[comp & 3u];
            px = ox + d.nx * sd; py = oy + d.ny * sd; pz = oz + d.nz * sd;
            excluded = 0xFFFFFFFFu;
            umax = 1.0f; umin = 0.0f;
            sub_n = 0;
            fresh = false;
        }
        const bool open = active;
        bool found;
        FastHit best;
        local_round<LAYOUT>(H, Lw, g, acc, lane, open, gx, gy, gz, ox, oy, oz, px, py, pz, excluded, found, best, pc);
        if (open) {
            bool finish = !found;
            if (found) {
                apply_hit(g, best, u, J.perm, J.reflType, umax, umin, ox, oy, oz, px, py, pz, comp, fiber, excluded,
                          nrefl, nperm);
                if (++sub_n >= J.maxSub) {
                    st |= kStatusSubsegCap;
                    px = ox; py = oy; pz = oz;
                    finish = true;
                }
            }
            if (finish) {
                // clamp in absolute coordinates, then move the origin so the
                // offset is back in [0, 1/16)
                float ax = gx + px, ay = gy + py, az = gz + pz;
                if (ax > J.clampHi) px = J.clampHi - gx; else if (ax < J.clampLo) px = J.clampLo - gx;
                if (ay > J.clampHi) py = J.clampHi - gy; else if (ay < J.clampLo) py = J.clampLo - gy;
                if (az > J.clampHi) pz = J.clampHi - gz; else if (az < J.clampLo) pz = J.clampLo - gz;
                const float sx = floor_small(px * 16.0f) * kLatticeH, sy = floor_small(py * 16.0f) * kLatticeH,
                            sz = floor_small(pz * 16.0f) * kLatticeH;
                gx += sx; gy += sy; gz += sz;
                ox = px - sx; oy = py - sy; oz = pz - sz;
                const float T2 = J.T2[comp & 3u];
                if (T2 > 0.0f) mag += -mag / T2 * J.dt;
                const float w = __ldg(J.wave + ls0 + it);
                kahan_add(mom[0][tx], mom[3][tx], w * (gx + ox));
                kahan_add(mom[1][tx], mom[4][tx], w * (gy + oy));
                kahan_add(mom[2][tx], mom[5][tx], w * (gz + oz));
                if (++it >= nsteps) active = false;
                else fresh = true;
            }
        }
        __syncwarp();
    }
    if (valid) {
        const double X = (double)gx + (double)ox, Y = (double)gy + (double)oy, Z = (double)gz + (double)oz;
        S.d[D_X][i] = X; S.d[D_Y][i] = Y; S.d[D_Z][i] = Z; S.d[D_MAG][i] = (double)mag;
        S.f[F_X][i] = (float)X; S.f[F_Y][i] = (float)Y; S.f[F_Z][i] = (float)Z;
        S.f[F_MAG][i] = mag;
        S.f[F_MX][i] = mom[0][tx]; S.f[F_MY][i] = mom[1][tx]; S.f[F_MZ][i] = mom[2][tx];
        S.f[F_CX][i] = mom[3][tx]; S.f[F_CY][i] = mom[4][tx]; S.f[F_CZ][i] = mom[5][tx];
        S.u[U_META][i] = (comp & 0xFFu) | (fiber << 8);
    }
    // per-job counters {reflections, permeations, records examined, FP64 re-tests}
    unsigned long long r = nrefl, p = nperm, te = pc.records, ex = pc.exact;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        r += __shfl_down_sync(FULL, r, o);
        p += __shfl_down_sync(FULL, p, o);
        te += __shfl_down_sync(FULL, te, o);
        ex += __shfl_down_sync(FULL, ex, o);
    }
    if (lane == 0) {
        if (r) atomicAdd(jobCounts + 4 * jb, r);
        if (p) atomicAdd(jobCounts + 4 * jb + 1, p);
        if (te) atomicAdd(jobCounts + 4 * jb + 2, te);
        if (ex) atomicAdd(jobCounts + 4 * jb + 3, ex);
    }
    if (st) atomicOr(status, st);
}

// LaneState of the FP64 form
struct LaneState64 {
    double mag[32], m[3][32], umax[32], umin[32], u[32], T2[32], rT2[32];
    uint32_t comp[32], fiber[32], nrefl[32], nperm[32], status[32], it[32], sub[32], decayOf[32];
};

// Precision-form mesh jobs (DSIM_JOB_PRECISE): the step of cpuIntegrate
// (dSim3/src/spinKernelCpu.cpp:430-499) in FP64 -- position, sub-segments,
// hits and reflections (prec_round.cuh), the clamp to +-(1 - spinRadius), the
// T2 decay and the gradient moments M += w(t) pos(t) -- on the same Philox
// draws as the plain form.  Positions and magnitudes persist in the double
// fields; the float fields receive their rounded values (sort keys, float
// readers) and the moment pair (m, c) holds M as m - c.
// Thin jobs at 3 blocks per SM (162 registers): two of them, all that such a job
// gives an SM, leave room beside them for the blocks of a cylinder job in the same
// launch; full warps at 4 (128).  ms of runs at 2 / 3 / 4: two jobs of 15,747 mesh
// and 13,586 cylinder spins 8.2 / 8.2 / 9.0 (9.0 with 198 registers), two of 32,768
// 7.0 / 7.0 / 7.2, six of 32,768 (full warps) 22.4 / 22.3 / 21.2.
template <int MINB>
__global__ void __launch_bounds__(kFlatThreads, MINB)
k_batch_step64(const SubDev* __restrict__ subs, const JobDev* __restrict__ jobs, BatchSpins S, StepWarps W,
               const uint32_t* __restrict__ stepNow, uint32_t chunk, uint32_t* status,
               unsigned long long* jobCounts) {
    __shared__ HitWarp wh[kFlatWarps];
    __shared__ PrecWarp wp[kFlatWarps];
    __shared__ LaneState64 wc[kFlatWarps];
    __shared__ JobDev jobS[kFlatWarps];
    __shared__ SubDev subS[kFlatWarps];
    const uint32_t FULL = 0xFFFFFFFFu;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t wi = threadIdx.x >> 5;
    HitWarp& H = wh[wi];
    PrecWarp& P = wp[wi];
    const uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (w >= W.count) return;  // whole warp
    const WarpSlots mine = warp_slots(W, w);
    const uint32_t i = mine.slot(lane);
    const uint32_t jb = S.u[U_JOB][mine.first];
    {
        const uint32_t* src = reinterpret_cast<const uint32_t*>(jobs + jb);
        uint32_t* dst = reinterpret_cast<uint32_t*>(jobS + wi);
        for (uint32_t k = lane; k < sizeof(JobDev) / 4; k += 32) dst[k] = __ldg(src + k);
        __syncwarp();
        const uint32_t* s2 = reinterpret_cast<const uint32_t*>(subs + jobS[wi].sub);
        uint32_t* d2 = reinterpret_cast<uint32_t*>(subS + wi);
        for (uint32_t k = lane; k < sizeof(SubDev) / 4; k += 32) d2[k] = __ldg(s2 + k);
        __syncwarp();
    }
    const JobDev& J = jobS[wi];
    const uint32_t now = *stepNow;
    const uint32_t start = J.start, steps = J.steps;
    if (now < start || now - start >= steps) return;
    const uint32_t ls0 = now - start;
    const uint32_t nsteps = min(chunk, steps - ls0);
    const uint32_t id = S.u[U_ID][i];
    const bool valid = id != 0xFFFFFFFFu && lane < mine.n;
    double ox = 0.0, oy = 0.0, oz = 0.0;
    LaneState64& C = wc[wi];
    double &mag = C.mag[lane], &Mx = C.m[0][lane], &My = C.m[1][lane], &Mz = C.m[2][lane], &umax = C.umax[lane],
           &umin = C.umin[lane], &u = C.u[lane], &T2 = C.T2[lane], &rT2 = C.rT2[lane];
    uint32_t &comp = C.comp[lane], &fiber = C.fiber[lane], &nrefl = C.nrefl[lane], &nperm = C.nperm[lane],
             &st = C.status[lane], &it = C.it[lane], &sub_n = C.sub[lane], &decayOf = C.decayOf[lane];
    mag = Mx = My = Mz = umin = T2 = rT2 = 0.0;
    u = umax = 1.0;
    comp = fiber = nrefl = nperm = st = it = sub_n = 0;
    decayOf = 4u;  // the compartment that T2 and rT2 are of
    if (valid) {
        ox = S.d[D_X][i]; oy = S.d[D_Y][i]; oz = S.d[D_Z][i]; mag = S.d[D_MAG][i];
        Mx = (double)S.f[F_MX][i] - (double)S.f[F_CX][i];
        My = (double)S.f[F_MY][i] - (double)S.f[F_CY][i];
        Mz = (double)S.f[F_MZ][i] - (double)S.f[F_CZ][i];
        const uint32_t meta = S.u[U_META][i];
        comp = meta & 0xFFu; fiber = meta >> 8;
    }
    const MeshDev& g = subS[wi].g;
    const AccelDev& acc = subS[wi].acc;
    const double perm = (double)J.perm;
    const double hiC = 1.0 - (double)J.spinR, loC = -1.0 + (double)J.spinR;
    // a point whose float coordinates keep inside this needs no clamp
    const float inside = (float)hiC - 1e-6f;
    const uint32_t reflType = J.reflType, maxSub = J.maxSub;
    const uint32_t k0 = J.key0, k1 = J.key1;
    const float* __restrict__ wave = J.wave;
    uint32_t excluded = 0xFFFFFFFFu;
    PrecCount pc;
    bool active = valid && nsteps > 0;
    bool fresh = active;
    // the position is o at the top of a step, the start of its current sub-segment within one
    double px = ox, py = oy, pz = oz;
    while (__any_sync(FULL, active)) {
        if (fresh) {
            const Draw d = philox_draw(id, (uint64_t)(ls0 + it), 0u, k0, k1);
            const double sd = (double)J.sd[comp & 3u];
            px = ox + (double)d.nx * sd; py = oy + (double)d.ny * sd; pz = oz + (double)d.nz * sd;
            u = (double)d.u;
            excluded = 0xFFFFFFFFu;
            umax = 1.0; umin = 0.0;
            sub_n = 0;
            fresh = false;
        }
        const bool open = active;
        bool found;
        uint32_t ht = 0, htype = 0;
        double hx = 0.0, hy = 0.0, hz = 0.0;
        prec_round(H, P, g, acc, lane, open, ox, oy, oz, px, py, pz, excluded, found, ht, htype, hx, hy, hz, pc);
        if (open) {
            bool finish = !found;
            if (found) {
                apply_hit64(g, ht, htype, hx, hy, hz, u, perm, reflType, umax, umin, ox, oy, oz, px, py, pz, comp,
                            fiber, excluded, nrefl, nperm);
                if (++sub_n >= maxSub) {
                    st |= kStatusSubsegCap;
                    px = ox; py = oy; pz = oz;
                    finish = true;
                }
            }
            if (finish) {
                if (!(fmaxf(fabsf((float)px), fmaxf(fabsf((float)py), fabsf((float)pz))) < inside)) {
                    if (px > hiC) px = hiC; else if (px < loC) px = loC;
                    if (py > hiC) py = hiC; else if (py < loC) py = loC;
                    if (pz > hiC) pz = hiC; else if (pz < loC) pz = loC;
                }
                ox = px; oy = py; oz = pz;
                if ((comp & 3u) != decayOf) {
                    decayOf = comp & 3u;
                    T2 = (double)J.T2[decayOf];
                    rT2 = 1.0 / T2;
                }
                if (T2 > 0.0) mag += div_by(-mag, T2, rT2) * (double)J.dt;
                const double w = (double)__ldg(wave + ls0 + it);
                Mx += w * ox; My += w * oy; Mz += w * oz;
                if (++it >= nsteps) active = false;
                else fresh = true;
            }
        }
        __syncwarp();
    }
    if (valid) {
        S.d[D_X][i] = ox; S.d[D_Y][i] = oy; S.d[D_Z][i] = oz; S.d[D_MAG][i] = mag;
        S.f[F_X][i] = (float)ox; S.f[F_Y][i] = (float)oy; S.f[F_Z][i] = (float)oz;
        S.f[F_MAG][i] = (float)mag;
        const float mx = (float)Mx, my = (float)My, mz = (float)Mz;
        S.f[F_MX][i] = mx; S.f[F_MY][i] = my; S.f[F_MZ][i] = mz;
        S.f[F_CX][i] = (float)((double)mx - Mx);
        S.f[F_CY][i] = (float)((double)my - My);
        S.f[F_CZ][i] = (float)((double)mz - Mz);
        S.u[U_META][i] = (comp & 0xFFu) | (fiber << 8);
    }
    // per-job counters {reflections, permeations, records examined, FP64 triangle tests}
    unsigned long long r = nrefl, p = nperm, te = pc.records, ex = pc.exact;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        r += __shfl_down_sync(FULL, r, o);
        p += __shfl_down_sync(FULL, p, o);
        te += __shfl_down_sync(FULL, te, o);
        ex += __shfl_down_sync(FULL, ex, o);
    }
    if (lane == 0) {
        if (r) atomicAdd(jobCounts + 4 * jb, r);
        if (p) atomicAdd(jobCounts + 4 * jb + 1, p);
        if (te) atomicAdd(jobCounts + 4 * jb + 2, te);
        if (ex) atomicAdd(jobCounts + 4 * jb + 3, ex);
    }
    if (st) atomicOr(status, st);
}

__global__ void k_batch_advance(uint32_t* stepNow, uint32_t chunk) { *stepNow += chunk; }

// sort key: job's base + Morton code of the spin's cell in a 2^bits grid over
// the box (mesh jobs), or region and scattered id (cylinder jobs); padding goes
// to the job's last key
__global__ void k_batch_keys(const JobDev* __restrict__ jobs, BatchSpins S, uint32_t* keys,
                             uint32_t* hist) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= S.N) return;
    const JobDev& J = jobs[S.u[U_JOB][i]];
    const uint32_t bits = J.sortBits, n = 1u << bits, id = S.u[U_ID][i];
    uint32_t key;
    if (id == 0xFFFFFFFFu) {
        key = J.sortBase + ((J.sortRegion ? 2u : 1u) << (3 * bits)) - 1u;
    } else if (J.sortRegion) {
        // cylinder jobs: a spin outside every fiber scans its cell's fiber
        // list, one inside tests its own fiber, so the two kinds go to
        // separate warps; within a kind the spins are spread by their ids.
        // Neighbours share the crowded cells: in Morton order a few warps held
        // most of the long steps and set a launch's time (FP64 form, kcycles a
        // step of a warp: mean 5.9, largest 21.5), while the fiber lists stay in
        // L1 in any order.  ms of runs in Morton order / spread: two FP64 jobs
        // 8.9 / 8.3, two of 32,768 spins 8.2 / 7.2, six local jobs of 65,536
        // 21.5 / 20.7, six plain ones 14.0 / 13.5.
        const uint32_t region = (S.u[U_META][i] & 0xFFu) >= 2u ? 1u : 0u;
        key = J.sortBase + (region << (3 * bits)) + ((id * 0x9E3779B1u) >> (32u - 3u * bits));
    } else {
        const float s = 0.5f * (float)n;
        uint32_t a = (uint32_t)fminf(fmaxf(floorf((S.f[F_X][i] + 1.0f) * s), 0.0f), (float)(n - 1));
        uint32_t b = (uint32_t)fminf(fmaxf(floorf((S.f[F_Y][i] + 1.0f) * s), 0.0f), (float)(n - 1));
        uint32_t c = (uint32_t)fminf(fmaxf(floorf((S.f[F_Z][i] + 1.0f) * s), 0.0f), (float)(n - 1));
        key = J.sortBase + morton3(a, b, c);
    }
    keys[i] = key;
    atomicAdd(hist + key, 1u);
}

__global__ void k_batch_scatter(BatchSpins S, BatchSpins D, const uint32_t* __restrict__ keys,
                                const uint32_t* __restrict__ start, uint32_t* cursor) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= S.N) return;
    const uint32_t k = keys[i];
    const uint32_t j = start[k] + atomicAdd(cursor + k, 1u);
#pragma unroll
    for (int f = 0; f < kBF; f++) D.f[f][j] = S.f[f][i];
#pragma unroll
    for (int u = 0; u < kBU; u++) D.u[u][j] = S.u[u][i];
    if (S.d[0]) {
#pragma unroll
        for (int f = 0; f < kBD; f++) D.d[f][j] = S.d[f][i];
    }
}

// compaction: slot i of a kept job moves to remapped slot; job index remapped
__global__ void k_batch_compact(BatchSpins S, BatchSpins D, const int32_t* __restrict__ jobMap,
                                const int64_t* __restrict__ slotShift) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= S.N) return;
    const uint32_t jb = S.u[U_JOB][i];
    const int32_t nj = jobMap[jb];
    if (nj < 0) return;
    const uint32_t j = (uint32_t)((int64_t)i + slotShift[jb]);
#pragma unroll
    for (int f = 0; f < kBF; f++) D.f[f][j] = S.f[f][i];
    D.u[U_META][j] = S.u[U_META][i];
    D.u[U_JOB][j] = (uint32_t)nj;
    D.u[U_ID][j] = S.u[U_ID][i];
    if (S.d[0]) {
#pragma unroll
        for (int f = 0; f < kBD; f++) D.d[f][j] = S.d[f][i];
    }
}

// a job's spins in spin order
__global__ void k_batch_gather(BatchSpins S, uint32_t slot0, uint32_t len, float* pos3, float* mag,
                               float* mom6, uint32_t* meta) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= len) return;
    const uint32_t i = slot0 + k;
    const uint32_t id = S.u[U_ID][i];
    if (id == 0xFFFFFFFFu) return;
    pos3[3 * id] = S.f[F_X][i]; pos3[3 * id + 1] = S.f[F_Y][i]; pos3[3 * id + 2] = S.f[F_Z][i];
    mag[id] = S.f[F_MAG][i];
    mom6[6 * id] = S.f[F_MX][i]; mom6[6 * id + 1] = S.f[F_MY][i]; mom6[6 * id + 2] = S.f[F_MZ][i];
    mom6[6 * id + 3] = S.f[F_CX][i]; mom6[6 * id + 4] = S.f[F_CY][i]; mom6[6 * id + 5] = S.f[F_CZ][i];
    meta[id] = S.u[U_META][i];
}

// a precision-form job's FP64 positions and magnitudes in spin order
__global__ void k_batch_gather64(BatchSpins S, uint32_t slot0, uint32_t len, double* pos3, double* mag) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= len) return;
    const uint32_t i = slot0 + k;
    const uint32_t id = S.u[U_ID][i];
    if (id == 0xFFFFFFFFu) return;
    pos3[3 * id] = S.d[D_X][i]; pos3[3 * id + 1] = S.d[D_Y][i]; pos3[3 * id + 2] = S.d[D_Z][i];
    mag[id] = S.d[D_MAG][i];
}

// ---- readout -------------------------------------------------------------------
// sin and cos of 2 pi k / kTrig, each in two parts (trig_table)
static constexpr uint32_t kTrig = 1024;
struct __align__(16) Trig {
    double s, c, sLo, cLo;
};

// sin and cos of the angle p.  n is the integer nearest p kTrig / 2 pi (adding
// and subtracting 1.5 * 2^52 rounds, and leaves n's low bits in the sum's), and
// r = p - n 2 pi / kTrig with the step in two parts, at most pi / kTrig: the
// angle's table entry for n and the Taylor polynomials of sin r to r^5 and
// cos r - 1 to r^4 (next terms below 6e-22 and 2e-18), joined by the addition
// theorem with the table's value added last.  With the phase's fused sum the
// error against 128 bits is no larger than that of sincos() of the separately
// rounded phase (phases to 0.1, 1, 10, 1000, rms: 3.2e-17, 3.8e-17, 1.8e-16,
// 1.7e-14 against 3.2e-17, 3.8e-17, 2.1e-16, 2.1e-14).  18 FP64 operations; sincos() takes about
// 30, and the FP64 pipe (1/64 of the FP32 rate) is the readout's bound.
// Beyond 2^40 (and for no number) sincos() itself.
__device__ __forceinline__ void sincos_table(double p, const Trig* __restrict__ table, double& s, double& c) {
    constexpr double kHi = 6.283185307179586232 / (double)kTrig, kLo = 2.4492935982947064e-16 / (double)kTrig;
    constexpr double kMagic = 6755399441055744.0;
    if (((uint32_t)__double2hiint(p) & 0x7FFFFFFFu) >= 0x42700000u) {
        sincos(p, &s, &c);
        return;
    }
    const double q = __fma_rn(p, 1.0 / kHi, kMagic);
    const Trig T = table[(uint32_t)__double2loint(q) & (kTrig - 1u)];
    const double n = __dsub_rn(q, kMagic);
    const double r = __fma_rn(-n, kLo, __fma_rn(-n, kHi, p));
    const double z = __dmul_rn(r, r);
    const double sr = __fma_rn(__fma_rn(z, 1.0 / 120.0, -1.0 / 6.0), __dmul_rn(r, z), r);
    const double cr = __dmul_rn(z, __fma_rn(z, 1.0 / 24.0, -0.5));  // cos r - 1
    s = __dadd_rn(T.s, __fma_rn(T.c, sr, __fma_rn(T.s, cr, T.sLo)));
    c = __dadd_rn(T.c, __fma_rn(-T.s, sr, __fma_rn(T.c, cr, T.cLo)));
}

// Readout of one job for nG gradients sharing its waveform.  Warp w takes the
// 32 gradients [32 (w % gw), 32 (w % gw) + 32) and the spins of segment w / gw
// (contiguous slots): each lane keeps its own gradient's sums in registers, so
// no per-gradient reduction across threads is needed.  32 spins at a time, each
// lane fetches one and puts its FP64 moments and magnitude in shared memory
// (one conversion per spin and warp), then all lanes take them in turn.
// partials[segment][gradient][15] = {X, Y, n} for all spins and per compartment,
// each summed in slot order; k_batch_signal_final adds the segments in a fixed
// order, so the result does not depend on the launch.  kg: gradients in units of
// the table's angle.  fp64: the job keeps FP64 positions and magnitudes
// (precision and cell-local forms), which the readout then uses.
//
// Bound by the FP64 pipe: 23 operations per spin and gradient where the first
// form took about 48 (the spin's conversions on every lane, sincos, two sums).
// 65,537 spins x 384 gradients: 2.43 -> 1.10 ms a call.
static constexpr int kSigThreads = 128;
struct SigWarp {
    double x[32], y[32], z[32], m[32];
    uint32_t comp[32];
};
__global__ void __launch_bounds__(kSigThreads) k_batch_signal(BatchSpins S, uint32_t slot0, uint32_t len,
                                                              const double* __restrict__ kg, uint32_t nG,
                                                              uint32_t gw, uint32_t nseg, uint32_t segLen,
                                                              double region, bool fp64,
                                                              const Trig* __restrict__ trig, double* partials) {
    __shared__ Trig table[kTrig];
    __shared__ SigWarp sw[kSigThreads / 32];
    for (uint32_t k = threadIdx.x; k < 2 * kTrig; k += kSigThreads)
        reinterpret_cast<double2*>(table)[k] = __ldg(reinterpret_cast<const double2*>(trig) + k);
    __syncthreads();
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31u;
    if (warp >= gw * nseg) return;  // whole warps
    SigWarp& W = sw[threadIdx.x >> 5];
    const uint32_t gi = (warp % gw) * 32u + lane, sg = warp / gw;
    const bool live = gi < nG;
    const double gx = live ? kg[3 * gi] : 0.0, gy = live ? kg[3 * gi + 1] : 0.0, gz = live ? kg[3 * gi + 2] : 0.0;
    double cX[4] = {0.0, 0.0, 0.0, 0.0}, cY[4] = {0.0, 0.0, 0.0, 0.0};
    uint32_t cn[4] = {0u, 0u, 0u, 0u};
    const uint32_t k0 = sg * segLen, k1 = min(len, k0 + segLen);
    for (uint32_t kb = k0; kb < k1; kb += 32) {
        const uint32_t i = slot0 + min(kb + lane, k1 - 1u);
        bool in = kb + lane < k1 && S.u[U_ID][i] != 0xFFFFFFFFu;
        if (in && region > 0.0) {  // dSim2's readout box (dSim2/src/spinSystem.cpp:944-978)
            const double x = fp64 ? S.d[D_X][i] : (double)S.f[F_X][i];
            const double y = fp64 ? S.d[D_Y][i] : (double)S.f[F_Y][i];
            const double z = fp64 ? S.d[D_Z][i] : (double)S.f[F_Z][i];
            in = x > -region && x < region && y > -region && y < region && z > -region && z < region;
        }
        const uint32_t some = __ballot_sync(0xFFFFFFFFu, in);
        __syncwarp();  // the previous spins have been read
        if (in) {
            const uint32_t at = __popc(some & ((1u << lane) - 1u));
            W.x[at] = (double)S.f[F_MX][i] - (double)S.f[F_CX][i];
            W.y[at] = (double)S.f[F_MY][i] - (double)S.f[F_CY][i];
            W.z[at] = (double)S.f[F_MZ][i] - (double)S.f[F_CZ][i];
            W.m[at] = fp64 ? S.d[D_MAG][i] : (double)S.f[F_MAG][i];
            W.comp[at] = S.u[U_META][i] & 3u;
        }
        __syncwarp();
        const uint32_t n = __popc(some);
        for (uint32_t k = 0; k < n; k++) {  // the same spin on every lane: warp-uniform branches
            const double m = W.m[k];
            const uint32_t comp = W.comp[k];
            double sn, cs;
            sincos_table(__fma_rn(gx, W.x[k], __fma_rn(gy, W.y[k], __dmul_rn(gz, W.z[k]))), table, sn, cs);
#pragma unroll
            for (uint32_t q = 0; q < 4; q++)
                if (comp == q) {
                    cX[q] = __fma_rn(m, cs, cX[q]);
                    cY[q] = __fma_rn(m, sn, cY[q]);
                    cn[q]++;
                }
        }
    }
    if (!live) return;
    double* o = partials + ((size_t)sg * nG + gi) * 15;
    o[0] = (cX[0] + cX[1]) + (cX[2] + cX[3]);
    o[1] = (cY[0] + cY[1]) + (cY[2] + cY[3]);
    o[2] = (double)(cn[0] + cn[1] + cn[2] + cn[3]);
#pragma unroll
    for (int q = 0; q < 4; q++) { o[3 + 3 * q] = cX[q]; o[4 + 3 * q] = cY[q]; o[5 + 3 * q] = (double)cn[q]; }
}

// Adds the segments: 32 consecutive values a block (coalesced), 16 slices of the
// segments added side by side and then in slice order.  One thread per value
// over all segments took 26 us a call.
__global__ void __launch_bounds__(512) k_batch_signal_final(const double* __restrict__ partials, uint32_t nb,
                                                            uint32_t nG, double* out) {
    __shared__ double sh[16][33];
    const uint32_t t = blockIdx.x * 32 + threadIdx.x;
    double v = 0.0;
    if (t < nG * 15)
        for (uint32_t b = threadIdx.y; b < nb; b += 16) v += partials[(size_t)b * nG * 15 + t];
    sh[threadIdx.y][threadIdx.x] = v;
    __syncthreads();
    if (threadIdx.y > 0 || t >= nG * 15) return;
    for (int k = 1; k < 16; k++) v += sh[k][threadIdx.x];
    out[t] = v;
}

}  // namespace dsim

using namespace dsim;

struct BatchBuf {
    float* f[kBF] = {};
    uint32_t* u[kBU] = {};
    double* d[kBD] = {};
};

struct BatchJob {
    uint32_t id;            // public job id
    JobDev d;
    uint32_t nSpins, pad;
    uint64_t slot0;
    float* wave = nullptr;  // device table
    double pc = 0.0;        // phase constant 2 pi gamma dt
    bool retired = false;
    uint64_t counts[2] = {0, 0};
};

// the step kernels: one per form and fine-grid record layout
enum StepKind {
    kStepMesh, kStepMeshFull, kStepCyl, kStepMeshLocal, kStepMeshLocalFull, kStepMesh64, kStepCyl64, kStepCylLocal,
    kStepKinds
};

struct dsim_batch {
    cudaStream_t st = nullptr;
    // the step kernels of a chunk (one per record layout and form) advance
    // disjoint jobs: they run side by side on these streams, forked from st
    // after the sort and joined before the step counter advances
    static constexpr int kSide = 6;
    cudaStream_t side[kSide] = {};
    cudaEvent_t forkEv = nullptr, joinEv[kSide] = {};
    uint64_t cap = 0;
    uint32_t jobCap = 0;
    BatchBuf buf[2];
    int cur = 0;
    uint64_t N = 0;
    std::vector<SubDev> subs;
    std::vector<const dsim_mesh*> meshes;  // per substrate (null for cylinders)
    std::vector<const dsim_cyl*> cylsHeld; // cylinder substrates added (released on free)
    SubDev* d_subs = nullptr;
    uint32_t subCap = 256;
    std::vector<BatchJob> jobs;            // packing order
    uint32_t nextId = 0;
    JobDev* d_jobs = nullptr;
    unsigned long long* d_counts = nullptr;
    uint32_t* d_status = nullptr;
    Trig* d_trig = nullptr;             // readout: sin and cos table
    double* d_sig = nullptr;               // readout scratch: gradients, partial sums, result (grows)
    size_t sigCap = 0;
    uint32_t* d_stepNow = nullptr;
    uint32_t stepNow = 0;                  // host mirror of *d_stepNow
    uint32_t* keys = nullptr;
    uint32_t *hist = nullptr, *hstart = nullptr, *scratch = nullptr;
    uint64_t keyCap = 0, K = 0;
    // 5 blocks per SM: ms of runs of 200 steps at 4 / 5 / 6 / 7 (half of the spins
    // in meshes, of 100 tubes): 131,072 spins 4.92 / 4.78 / 4.90 / 5.16; 393,216
    // 15.2 / 14.4 / 14.7 / 14.6; 983,040 31.1 / 29.6 / 29.1 / 30.2
    uint32_t chunk = 20, occupancy = 5, graphChunks = 8;
    bool chunkSet = false;  // dsim_batch_configure or the autotuner chose the chunk
    uint32_t blockThreads = kFlatThreads;  // block size of the plain step kernels (64, 128, 256)
    // the warps of each kind of step kernel, as uploaded: built from the
    // unfinished jobs
    uint2* d_warps = nullptr;
    size_t warpCap = 0;
    StepWarps kinds[kStepKinds] = {};
    uint32_t warpsAt = 0;     // stepNow when they were built
    bool warpsValid = false;
    cudaGraphExec_t exec = nullptr;
    bool graphValid = false;
    int graphCur = -1;
    uint64_t launches = 0, graphLaunches = 0, bytes = 0;
};

namespace {

int balloc(dsim_batch* b, void** p, size_t bytes) {
    *p = nullptr;
    cudaError_t e = cudaMalloc(p, bytes ? bytes : 16);
    if (e != cudaSuccess) {
        cudaGetLastError();
        set_last_error(kErrNoMem, "batch: cudaMalloc(%zu): %s", bytes, cudaGetErrorString(e));
        return kErrNoMem;
    }
    b->bytes += bytes;
    return kOk;
}

BatchSpins view(dsim_batch* b, int which) {
    BatchSpins S;
    for (int f = 0; f < kBF; f++) S.f[f] = b->buf[which].f[f];
    for (int u = 0; u < kBU; u++) S.u[u] = b->buf[which].u[u];
    for (int f = 0; f < kBD; f++) S.d[f] = b->buf[which].d[f];
    S.N = (uint32_t)b->N;
    return S;
}

uint32_t sort_bits(uint32_t n) {
    // about two spins per sort cell: 2^(3 bits) ~ n / 2, 3..7 bits per axis
    uint32_t bits = 3;
    while (bits < 7 && (1ull << (3 * (bits + 1))) <= (uint64_t)n / 2) bits++;
    return bits;
}

void invalidate_graph(dsim_batch* b) {
    if (b->exec) cudaGraphExecDestroy(b->exec);
    b->exec = nullptr;
    b->graphValid = false;
}

// recompute sort key bases in packing order and grow the histogram
int layout_keys(dsim_batch* b) {
    uint64_t K = 0, slot = 0;
    for (auto& j : b->jobs) {
        j.d.sortBase = (uint32_t)K;
        K += (j.d.sortRegion ? 2ull : 1ull) << (3 * j.d.sortBits);
        j.slot0 = slot;
        slot += j.pad;
    }
    if (K > 0xFFFFFFF0ull) { set_last_error(kErrTooLarge, "batch: sort key space too large"); return kErrTooLarge; }
    if (K > b->keyCap) {
        cudaFree(b->hist); cudaFree(b->hstart); cudaFree(b->scratch);
        b->hist = b->hstart = b->scratch = nullptr;
        uint64_t cap = std::max<uint64_t>(K, 1u << 16) * 2;
        int rc;
        if ((rc = balloc(b, (void**)&b->hist, cap * 4)) || (rc = balloc(b, (void**)&b->hstart, (cap + 1) * 4)) ||
            (rc = balloc(b, (void**)&b->scratch, scan_scratch_words((uint32_t)cap) * 4)))
            return rc;
        b->keyCap = cap;
    }
    b->K = K;
    return kOk;
}

int upload_jobs(dsim_batch* b) {
    std::vector<JobDev> h(b->jobs.size());
    for (size_t k = 0; k < b->jobs.size(); k++) h[k] = b->jobs[k].d;
    if (!h.empty()) DSIM_CUDA_TRY(cudaMemcpyAsync(b->d_jobs, h.data(), h.size() * sizeof(JobDev), cudaMemcpyHostToDevice, b->st));
    return kOk;
}

StepKind kind_of(const dsim_batch* b, const BatchJob& j) {
    const SubDev& s = b->subs[j.d.sub];
    const bool cyl = s.kind == kSubCyl, full = s.acc.wide == 2;
    if (j.d.flags & DSIM_JOB_PRECISE) return cyl ? kStepCyl64 : kStepMesh64;
    if (j.d.flags & DSIM_JOB_LOCAL) return cyl ? kStepCylLocal : (full ? kStepMeshLocalFull : kStepMeshLocal);
    return cyl ? kStepCyl : (full ? kStepMeshFull : kStepMesh);
}

bool job_finished(const dsim_batch* b, const BatchJob& j) {
    return b->stepNow >= j.d.start && b->stepNow - j.d.start >= j.d.steps;
}

// A launch of few steps, by a configured chunk: the warps' reading of their job and
// substrate and their strided slots are then most of it, so they are fewer and (but
// for FP64 steps) take neighbouring slots.  us of 48 steps of 300,000 mesh spins at
// chunks of 1 / 2 / 4 / 8 as long launches and so: 5132 / 3686 / 2897 / 2292 and 4034 /
// 3079 / 2561 / 2099; of 60 cell-local jobs of 400, mesh and cylinders: 3137 / 2046 /
// 1558 / 1059 and 2372 / 1644 / 1333 / 937.
bool short_launches(const dsim_batch* b) { return b->chunkSet && b->chunk <= 8; }

// Warps per SM below which a kind's warps hold fewer than 32 spins.  FP32 mesh, ms
// of runs at 12 / 16 / 20 / 24 (with as many cylinder spins beside them): six jobs
// of 4957 to 35,814 spins 11.5 / 10.8 / 10.0 / 10.9; one mesh job of 8192 spins 1.54 /
// 1.62 / 1.68 / 1.70, of 16,384 2.26 / 2.24 / 2.24 / 2.39, of 40,960 3.42 / 3.23 / 3.26 /
// 3.46, of 65,536 4.25 / 4.16 / 4.05 / 4.44.  The others, us per step at 32 / 16 / 8 /
// 4 / 2 spins a warp: cell-local mesh 16,384 spins 17.0 / 13.0 / 10.4 / 13.1, 32,768
// 18.8 / 14.7 / 18.5; FP64 mesh 4096 26.8 / 19.8 / 15.8 / 14.5 / 17.7, 16,384 32.3 /
// 28.7 / 31.6; FP32 cylinders 16,384 6.3 / 5.7 / 4.0 / 3.4 / 3.9, 49,152 8.5 / 6.7 / 5.8 /
// 6.3; cell-local cylinders 32,768 11.4 / 8.6 / 7.3 / 7.4; FP64 cylinders 4096 28.9 /
// 20.2 / 17.9 / 16.2 / 20.6, 32,768 48.5 / 46.7 / 52.3.
// No more than the configured blocks per SM hold at once: 60,000 FP32 mesh spins at 4
// blocks, launches of 48 steps, 626 us at 20 warps and 469 at 16.
uint32_t warps_per_sm(const dsim_batch* b, StepKind k) {
    if (short_launches(b)) return 8;
    switch (k) {
        case kStepCyl: case kStepCylLocal: return 41;
        case kStepMesh64: case kStepCyl64: return 8;
        case kStepMesh: case kStepMeshFull: return std::min(20u, 4u * b->occupancy);
        default: return 16;
    }
}
uint32_t spins_per_warp_of(const dsim_batch* b, StepKind k, uint64_t spins) {
    return spins_per_warp(spins, warps_per_sm(b, k), k == kStepCyl || k == kStepCylLocal || k == kStepCyl64);
}

// lists the warps of the unfinished jobs by kind
int build_warps(dsim_batch* b) {
    std::vector<uint2> list;
    size_t first[kStepKinds];
    uint64_t spins[kStepKinds] = {};
    for (const auto& j : b->jobs)
        if (!job_finished(b, j)) spins[kind_of(b, j)] += j.nSpins;
    for (int k = 0; k < kStepKinds; k++) {
        first[k] = list.size();
        const uint32_t per = spins_per_warp_of(b, (StepKind)k, spins[k]);
        for (const auto& j : b->jobs) {
            if (job_finished(b, j) || kind_of(b, j) != (StepKind)k) continue;
            const uint32_t warps = (j.pad + per - 1) / per;
            const bool deal = k == kStepMesh64 || (k != kStepCyl && k != kStepCyl64 && k != kStepCylLocal && !short_launches(b));
            for (uint32_t w = 0; w < warps; w++) {
                // w0: the first of the warps that share slots, `dealt` of them, n slots in all
                const uint32_t w0 = deal ? w / kDealWarps * kDealWarps : w, dealt = deal ? std::min(kDealWarps, warps - w0) : 1u;
                const uint32_t n = std::min(j.pad - w0 * per, dealt * per), q = w - w0;
                list.push_back(make_uint2((uint32_t)j.slot0 + w0 * per + q, (n - q + dealt - 1) / dealt | dealt << 8));
            }
        }
        b->kinds[k].count = (uint32_t)(list.size() - first[k]);
        b->kinds[k].per = per;
    }
    if (list.size() > b->warpCap) {
        cudaFree(b->d_warps);
        b->bytes -= b->warpCap * sizeof(uint2);
        b->d_warps = nullptr; b->warpCap = 0;
        const size_t cap = std::max<size_t>(list.size() * 2, 1024);
        int rc = balloc(b, (void**)&b->d_warps, cap * sizeof(uint2));
        if (rc) return rc;
        b->warpCap = cap;
    }
    for (int k = 0; k < kStepKinds; k++) b->kinds[k].warp = b->d_warps + first[k];
    if (!list.empty())
        DSIM_CUDA_TRY(cudaMemcpyAsync(b->d_warps, list.data(), list.size() * sizeof(uint2), cudaMemcpyHostToDevice, b->st));
    b->warpsAt = b->stepNow;
    b->warpsValid = true;
    invalidate_graph(b);
    return kOk;
}

// builds them when jobs came or went, or when so many have finished that a
// kind's warps should hold at most three quarters of the spins they do
int ensure_warps(dsim_batch* b) {
    bool stale = !b->warpsValid;
    if (!stale && b->warpsAt != b->stepNow) {
        uint64_t left[kStepKinds] = {};
        for (const auto& j : b->jobs)
            if (!job_finished(b, j)) left[kind_of(b, j)] += j.nSpins;
        for (int k = 0; k < kStepKinds; k++)
            stale = stale || (b->kinds[k].count > 0 &&
                              (left[k] == 0 || 4 * spins_per_warp_of(b, (StepKind)k, left[k]) <= 3 * b->kinds[k].per));
    }
    return stale ? build_warps(b) : kOk;
}

// kernels one chunk launches: keys, scan (3), scatter, the step kernels, advance
uint64_t chunk_launches(const dsim_batch* b) {
    uint64_t n = 6;
    for (const StepWarps& W : b->kinds) n += W.count > 0;
    return n;
}

// Precision-form cylinder jobs (DSIM_JOB_PRECISE): the dSim2 step of
// cpuIntegrate (dSim2/src/spinKernelCpu.cpp:312-641) with positions,
// distances, clamp, T2 decay and moments in double (cyl_membranes); the
// parameters are the job's float values.  Position and magnitude persist in
// the double fields; the moment is kept as the float pair m - c.
__global__ void __launch_bounds__(kFlatThreads, 4)
k_batch_step_cyl64(const SubDev* __restrict__ subs, const JobDev* __restrict__ jobs, BatchSpins S, StepWarps W,
                   const uint32_t* __restrict__ stepNow, uint32_t chunk, uint32_t* status,
                   unsigned long long* jobCounts) {
    const uint32_t FULL = 0xFFFFFFFFu;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (w >= W.count) return;  // whole warp
    const WarpSlots mine = warp_slots(W, w);
    const uint32_t at = lane & (W.per - 1u), i = mine.slot(at);  // the lanes repeat the spins
    const uint32_t jb = S.u[U_JOB][mine.first];
    const JobDev& J = jobs[jb];
    const SubDev& sub = subs[__ldg(&J.sub)];
    const uint32_t now = *stepNow;
    const uint32_t start = __ldg(&J.start), steps = __ldg(&J.steps);
    if (now < start || now - start >= steps) return;
    const uint32_t ls0 = now - start;
    const uint32_t nsteps = min(chunk, steps - ls0);
    const uint32_t id = S.u[U_ID][i];
    const bool valid = id != 0xFFFFFFFFu && at < mine.n;
    const uint32_t live = __ballot_sync(FULL, valid);  // ThinDraws
    uint32_t nrefl = 0, nperm = 0, st = 0;
    if (valid) {
        ThinDraws draws;
        const CylDev g = sub.c;
        double x = S.d[D_X][i], y = S.d[D_Y][i], z = S.d[D_Z][i], mag = S.d[D_MAG][i];
        double Mx = (double)S.f[F_MX][i] - (double)S.f[F_CX][i];
        double My = (double)S.f[F_MY][i] - (double)S.f[F_CY][i];
        double Mz = (double)S.f[F_MZ][i] - (double)S.f[F_CZ][i];
        const uint32_t meta = S.u[U_META][i];
        uint32_t imo = meta & 0xFFu, nearest = meta >> 8;
        if (imo < 2 && nearest >= g.nF) imo = 2;
        const double perm = (double)__ldg(&J.perm);
        Cyl64 form = {(double)__ldg(&J.inR)};
        bool clear = false;
        const double hiC = 1.0 - (double)__ldg(&J.spinR), loC = -1.0 + (double)__ldg(&J.spinR);
        // a point whose float coordinates keep inside this needs no clamp
        const float inside = (float)hiC - 1e-6f;
        const double dt = (double)__ldg(&J.dt);
        const uint32_t k0 = __ldg(&J.key0), k1 = __ldg(&J.key1);
        const float* __restrict__ wave = J.wave;
        uint32_t decayOf = 3u;  // the region that T2 and rT2 are of
        double T2 = 0.0, rT2 = 0.0;
        for (uint32_t it = 0; it < nsteps; it++) {
            const Draw d = draws.step(it, W.per, lane, live, id, ls0, k0, k1);
            const double sd = (double)__ldg(&J.sd[imo == 0 ? 0 : (imo == 1 ? 1 : 2)]);
            const P3<double> o = {x, y, z};
            P3<double> p = {x + (double)d.nx * sd, y + (double)d.ny * sd, z + (double)d.nz * sd};
            cyl_membranes(g, form, o, p, (double)d.u, perm, imo, nearest, nrefl, nperm, st, clear);
            if (!(fmaxf(fabsf((float)p.x), fmaxf(fabsf((float)p.y), fabsf((float)p.z))) < inside))
                cyl_clamp(p, loC, hiC, clear);
            x = p.x; y = p.y; z = p.z;
            if (imo <= 2) {
                if (imo != decayOf) {
                    decayOf = imo;
                    T2 = (double)__ldg(&J.T2[imo]);
                    rT2 = 1.0 / T2;
                }
                if (T2 > 0.0) mag += div_by(-mag, T2, rT2) * dt;
            }
            const double w = (double)__ldg(wave + ls0 + it);
            Mx += w * x; My += w * y; Mz += w * z;
        }
        if (lane == at) {
            S.d[D_X][i] = x; S.d[D_Y][i] = y; S.d[D_Z][i] = z; S.d[D_MAG][i] = mag;
            S.f[F_X][i] = (float)x; S.f[F_Y][i] = (float)y; S.f[F_Z][i] = (float)z;
            S.f[F_MAG][i] = (float)mag;
            const float mx = (float)Mx, my = (float)My, mz = (float)Mz;
            S.f[F_MX][i] = mx; S.f[F_MY][i] = my; S.f[F_MZ][i] = mz;
            S.f[F_CX][i] = (float)((double)mx - Mx);
            S.f[F_CY][i] = (float)((double)my - My);
            S.f[F_CZ][i] = (float)((double)mz - Mz);
            S.u[U_META][i] = (imo & 0xFFu) | ((nearest & 0xFFFFFFu) << 8);
        } else {
            nrefl = nperm = 0;  // counted once
        }
    }
    unsigned long long r = nrefl, p = nperm;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        r += __shfl_down_sync(FULL, r, o);
        p += __shfl_down_sync(FULL, p, o);
    }
    if (lane == 0) {
        if (r) atomicAdd(jobCounts + 4 * jb, r);
        if (p) atomicAdd(jobCounts + 4 * jb + 1, p);
    }
    if (st) atomicOr(status, st);
}

// Cell-local FP32 cylinder jobs (DSIM_JOB_LOCAL): the dSim2 step with the
// position as a lattice origin (multiple of 1/16) plus an FP32 offset in
// [0, 1/16), membrane decisions near their FP32 error band taken in FP64
// (CylLocal), Kahan moments.  Between chunks the position is kept
// in the double fields as origin + offset.
__global__ void __launch_bounds__(kFlatThreads, 4)
k_batch_step_cyl_local(const SubDev* __restrict__ subs, const JobDev* __restrict__ jobs, BatchSpins S, StepWarps W,
                       const uint32_t* __restrict__ stepNow, uint32_t chunk, uint32_t* status,
                       unsigned long long* jobCounts) {
    __shared__ float mom[6][kFlatThreads];
    const uint32_t FULL = 0xFFFFFFFFu;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t tx = threadIdx.x;
    const uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (w >= W.count) return;  // whole warp
    const WarpSlots mine = warp_slots(W, w);
    const uint32_t at = lane & (W.per - 1u), i = mine.slot(at);  // the lanes repeat the spins
    const uint32_t jb = S.u[U_JOB][mine.first];
    const JobDev& J = jobs[jb];
    const SubDev& sub = subs[__ldg(&J.sub)];
    const uint32_t now = *stepNow;
    const uint32_t start = __ldg(&J.start), steps = __ldg(&J.steps);
    if (now < start || now - start >= steps) return;
    const uint32_t ls0 = now - start;
    const uint32_t nsteps = min(chunk, steps - ls0);
    const uint32_t id = S.u[U_ID][i];
    const bool valid = id != 0xFFFFFFFFu && at < mine.n;
    const uint32_t live = __ballot_sync(FULL, valid);  // ThinDraws
    uint32_t nrefl = 0, nperm = 0, st = 0;
    CylLocal form = {__ldg(&J.inR), {0.0f, 0.0f, 0.0f}, 0u, 0u};
    if (valid) {
        ThinDraws draws;
        const CylDev g = sub.c;
        const double X = S.d[D_X][i], Y = S.d[D_Y][i], Z = S.d[D_Z][i];
        CylOrigin& G = form.G;
        G.x = (float)(floor(X * 16.0) * 0.0625);
        G.y = (float)(floor(Y * 16.0) * 0.0625);
        G.z = (float)(floor(Z * 16.0) * 0.0625);
        float x = (float)(X - (double)G.x), y = (float)(Y - (double)G.y), z = (float)(Z - (double)G.z);
        float mag = S.f[F_MAG][i];
        mom[0][tx] = S.f[F_MX][i]; mom[1][tx] = S.f[F_MY][i]; mom[2][tx] = S.f[F_MZ][i];
        mom[3][tx] = S.f[F_CX][i]; mom[4][tx] = S.f[F_CY][i]; mom[5][tx] = S.f[F_CZ][i];
        const uint32_t meta = S.u[U_META][i];
        uint32_t imo = meta & 0xFFu, nearest = meta >> 8;
        if (imo < 2 && nearest >= g.nF) imo = 2;
        const float perm = __ldg(&J.perm);
        bool clear = false;
        const float clampHi = __ldg(&J.clampHi), clampLo = __ldg(&J.clampLo), dt = __ldg(&J.dt);
        const uint32_t k0 = __ldg(&J.key0), k1 = __ldg(&J.key1);
        const float* __restrict__ wave = J.wave;
        for (uint32_t it = 0; it < nsteps; it++) {
            const Draw d = draws.step(it, W.per, lane, live, id, ls0, k0, k1);
            const float sd = __ldg(&J.sd[imo < 3 ? imo : 2]);
            const P3<float> o = {x, y, z};
            P3<float> p = {x + d.nx * sd, y + d.ny * sd, z + d.nz * sd};
            cyl_membranes(g, form, o, p, d.u, perm, imo, nearest, nrefl, nperm, st, clear);
            // clamp in absolute coordinates, then move the origin so the
            // offset is back in [0, 1/16)
            const P3<float> q = p;
            if (G.x + p.x > clampHi) p.x = clampHi - G.x; else if (G.x + p.x < clampLo) p.x = clampLo - G.x;
            if (G.y + p.y > clampHi) p.y = clampHi - G.y; else if (G.y + p.y < clampLo) p.y = clampLo - G.y;
            if (G.z + p.z > clampHi) p.z = clampHi - G.z; else if (G.z + p.z < clampLo) p.z = clampLo - G.z;
            clear = clear & (p.x == q.x) & (p.y == q.y) & (p.z == q.z);
            const float sx = floor_small(p.x * 16.0f) * kLatticeH, sy = floor_small(p.y * 16.0f) * kLatticeH,
                        sz = floor_small(p.z * 16.0f) * kLatticeH;
            G.x += sx; G.y += sy; G.z += sz;
            x = p.x - sx; y = p.y - sy; z = p.z - sz;
            const float T2 = __ldg(&J.T2[imo < 3 ? imo : 2]);
            if (T2 > 0.0f) mag += -mag / T2 * dt;
            const float w = __ldg(wave + ls0 + it);
            kahan_add(mom[0][tx], mom[3][tx], w * (G.x + x));
            kahan_add(mom[1][tx], mom[4][tx], w * (G.y + y));
            kahan_add(mom[2][tx], mom[5][tx], w * (G.z + z));
        }
        const double Xn = (double)G.x + (double)x, Yn = (double)G.y + (double)y, Zn = (double)G.z + (double)z;
        if (lane == at) {
            S.d[D_X][i] = Xn; S.d[D_Y][i] = Yn; S.d[D_Z][i] = Zn; S.d[D_MAG][i] = (double)mag;
            S.f[F_X][i] = (float)Xn; S.f[F_Y][i] = (float)Yn; S.f[F_Z][i] = (float)Zn;
            S.f[F_MAG][i] = mag;
            S.f[F_MX][i] = mom[0][tx]; S.f[F_MY][i] = mom[1][tx]; S.f[F_MZ][i] = mom[2][tx];
            S.f[F_CX][i] = mom[3][tx]; S.f[F_CY][i] = mom[4][tx]; S.f[F_CZ][i] = mom[5][tx];
            S.u[U_META][i] = (imo & 0xFFu) | ((nearest & 0xFFFFFFu) << 8);
        } else {
            nrefl = nperm = form.ntests = form.nexact = 0;  // counted once
        }
    }
    // per-job counters {reflections, permeations, distance tests, FP64 decisions}
    unsigned long long r = nrefl, p = nperm, te = form.ntests, ex = form.nexact;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        r += __shfl_down_sync(FULL, r, o);
        p += __shfl_down_sync(FULL, p, o);
        te += __shfl_down_sync(FULL, te, o);
        ex += __shfl_down_sync(FULL, ex, o);
    }
    if (lane == 0) {
        if (r) atomicAdd(jobCounts + 4 * jb, r);
        if (p) atomicAdd(jobCounts + 4 * jb + 1, p);
        if (te) atomicAdd(jobCounts + 4 * jb + 2, te);
        if (ex) atomicAdd(jobCounts + 4 * jb + 3, ex);
    }
    if (st) atomicOr(status, st);
}

uint32_t step_grid(const StepWarps& W, int threads) {
    return (uint32_t)(((uint64_t)W.count * 32 + threads - 1) / threads);
}

template <int LAYOUT, int THREADS>
void launch_step_shape(dsim_batch* b, const BatchSpins& D, const StepWarps& W, uint32_t steps, cudaStream_t st) {
    const uint32_t grid = step_grid(W, THREADS);
    if (b->occupancy >= 8)
        k_batch_step<8, LAYOUT, THREADS><<<grid, THREADS, 0, st>>>(b->d_subs, b->d_jobs, D, W, b->d_stepNow, steps,
                                                                  b->d_status, b->d_counts);
    else if (b->occupancy >= 6)
        k_batch_step<6, LAYOUT, THREADS><<<grid, THREADS, 0, st>>>(b->d_subs, b->d_jobs, D, W, b->d_stepNow, steps,
                                                                  b->d_status, b->d_counts);
    else if (b->occupancy == 5)
        k_batch_step<5, LAYOUT, THREADS><<<grid, THREADS, 0, st>>>(b->d_subs, b->d_jobs, D, W, b->d_stepNow, steps,
                                                                  b->d_status, b->d_counts);
    else
        k_batch_step<4, LAYOUT, THREADS><<<grid, THREADS, 0, st>>>(b->d_subs, b->d_jobs, D, W, b->d_stepNow, steps,
                                                                  b->d_status, b->d_counts);
}

template <int LAYOUT>
void launch_step_layout(dsim_batch* b, const BatchSpins& D, const StepWarps& W, uint32_t steps, cudaStream_t st) {
    if (b->blockThreads == 64) launch_step_shape<LAYOUT, 64>(b, D, W, steps, st);
    else if (b->blockThreads == 256) launch_step_shape<LAYOUT, 256>(b, D, W, steps, st);
    else launch_step_shape<LAYOUT, kFlatThreads>(b, D, W, steps, st);
}

// sort into the other buffer, `steps` steps, advance the step counter; the
// warps are current (ensure_warps)
int enqueue_chunk(dsim_batch* b, uint32_t steps) {
    const uint32_t N = (uint32_t)b->N;
    const uint32_t nb = (N + 255) / 256;
    BatchSpins S = view(b, b->cur), D = view(b, 1 - b->cur);
    DSIM_CUDA_TRY(cudaMemsetAsync(b->hist, 0, b->K * 4, b->st));
    k_batch_keys<<<nb, 256, 0, b->st>>>(b->d_jobs, S, b->keys, b->hist);
    int rc = launch_scan_exclusive(b->hist, b->hstart, (uint32_t)b->K, b->scratch, b->st);
    if (rc) return rc;
    DSIM_CUDA_TRY(cudaMemsetAsync(b->hist, 0, b->K * 4, b->st));
    k_batch_scatter<<<nb, 256, 0, b->st>>>(S, D, b->keys, b->hstart, b->hist);
    b->cur = 1 - b->cur;
    // the step kernels this chunk needs, each on its own stream when there
    // are several (they advance disjoint jobs)
    int kinds[kStepKinds], nk = 0;
    for (int k = 0; k < kStepKinds; k++)
        if (b->kinds[k].count > 0) kinds[nk++] = k;
    const bool fork = nk > 1;
    if (fork) DSIM_CUDA_TRY(cudaEventRecord(b->forkEv, b->st));
    for (int q = 0; q < nk; q++) {
        cudaStream_t st = fork ? b->side[q % dsim_batch::kSide] : b->st;
        if (fork) DSIM_CUDA_TRY(cudaStreamWaitEvent(st, b->forkEv, 0));
        const StepWarps& W = b->kinds[kinds[q]];
        const uint32_t grid = step_grid(W, kFlatThreads);
        switch (kinds[q]) {
            case kStepMesh: launch_step_layout<1>(b, D, W, steps, st); break;
            case kStepMeshFull: launch_step_layout<2>(b, D, W, steps, st); break;
            case kStepCyl: launch_step_layout<3>(b, D, W, steps, st); break;
            case kStepMeshLocal:
                k_batch_step_local<1><<<grid, kFlatThreads, 0, st>>>(b->d_subs, b->d_jobs, D, W, b->d_stepNow, steps,
                                                                     b->d_status, b->d_counts);
                break;
            case kStepMeshLocalFull:
                k_batch_step_local<2><<<grid, kFlatThreads, 0, st>>>(b->d_subs, b->d_jobs, D, W, b->d_stepNow, steps,
                                                                     b->d_status, b->d_counts);
                break;
            case kStepMesh64:
                if (W.per < 32)
                    k_batch_step64<3><<<grid, kFlatThreads, 0, st>>>(b->d_subs, b->d_jobs, D, W, b->d_stepNow, steps,
                                                                     b->d_status, b->d_counts);
                else
                    k_batch_step64<4><<<grid, kFlatThreads, 0, st>>>(b->d_subs, b->d_jobs, D, W, b->d_stepNow, steps,
                                                                     b->d_status, b->d_counts);
                break;
            case kStepCyl64:
                k_batch_step_cyl64<<<grid, kFlatThreads, 0, st>>>(b->d_subs, b->d_jobs, D, W, b->d_stepNow, steps,
                                                                  b->d_status, b->d_counts);
                break;
            default:
                k_batch_step_cyl_local<<<grid, kFlatThreads, 0, st>>>(b->d_subs, b->d_jobs, D, W, b->d_stepNow, steps,
                                                                      b->d_status, b->d_counts);
                break;
        }
        if (fork) {
            DSIM_CUDA_TRY(cudaEventRecord(b->joinEv[q % dsim_batch::kSide], st));
            DSIM_CUDA_TRY(cudaStreamWaitEvent(b->st, b->joinEv[q % dsim_batch::kSide], 0));
        }
    }
    k_batch_advance<<<1, 1, 0, b->st>>>(b->d_stepNow, steps);
    DSIM_CUDA_TRY(cudaGetLastError());
    b->launches += chunk_launches(b);
    return kOk;
}

int capture_graph(dsim_batch* b) {
    invalidate_graph(b);
    const uint32_t G = b->graphChunks & ~1u;  // even: the buffers end where they start
    if (G == 0) return kOk;
    const int cur0 = b->cur;
    const uint64_t launches0 = b->launches;
    cudaGraph_t graph = nullptr;
    DSIM_CUDA_TRY(cudaStreamBeginCapture(b->st, cudaStreamCaptureModeThreadLocal));
    int rc = kOk;
    for (uint32_t c = 0; c < G && !rc; c++) rc = enqueue_chunk(b, b->chunk);
    cudaError_t e = cudaStreamEndCapture(b->st, &graph);
    b->cur = cur0;
    b->launches = launches0;
    if (rc) { if (graph) cudaGraphDestroy(graph); return rc; }
    if (e != cudaSuccess) { set_last_cuda_error(e, "cudaStreamEndCapture", __FILE__, __LINE__); return kErrCuda; }
    e = cudaGraphInstantiate(&b->exec, graph, 0);
    cudaGraphDestroy(graph);
    if (e != cudaSuccess) { b->exec = nullptr; set_last_cuda_error(e, "cudaGraphInstantiate", __FILE__, __LINE__); return kErrCuda; }
    b->graphValid = true;
    b->graphCur = cur0;
    return kOk;
}

BatchJob* find_job(dsim_batch* b, uint32_t id) {
    for (auto& j : b->jobs)
        if (j.id == id) return &j;
    return nullptr;
}

constexpr double kPi = 3.14159265358979323846;

// the readout's table, made once: the nearest doubles and what they leave
// (long double has 64 bits of significand or more here)
const Trig* trig_table() {
    static const std::vector<Trig> table = [] {
        std::vector<Trig> t(kTrig);
        for (uint32_t k = 0; k < kTrig; k++) {
            const long double a = 6.283185307179586476925286766559L * (long double)k / (long double)kTrig;
            const long double s = sinl(a), c = cosl(a);
            t[k].s = (double)s; t[k].c = (double)c;
            t[k].sLo = (double)(s - (long double)t[k].s); t[k].cLo = (double)(c - (long double)t[k].c);
        }
        return t;
    }();
    return table.data();
}

std::vector<float> make_wave(const dsim_job_desc* d) {
    std::vector<float> w(d->steps, 0.0f);
    if (d->waveform == DSIM_WAVE_TABLE) {
        for (uint32_t s = 0; s < d->steps; s++) w[s] = d->table[s];
        return w;
    }
    const long nd = lround((double)d->delta / (double)d->deltaTime);
    const long nD = lround((double)d->Delta / (double)d->deltaTime);
    for (uint32_t s = 0; s < d->steps; s++) {
        const long t = (long)s;
        if (t < nd) {
            w[s] = d->waveform == DSIM_WAVE_OGSE
                       ? (float)std::cos(2.0 * kPi * (double)d->frequency * 1e-3 * (double)t * (double)d->deltaTime)
                       : 1.0f;
        } else if (t >= nD && t < nD + nd) {
            w[s] = d->waveform == DSIM_WAVE_OGSE
                       ? -(float)std::cos(2.0 * kPi * (double)d->frequency * 1e-3 * (double)(t - nD) * (double)d->deltaTime)
                       : -1.0f;
        }
    }
    return w;
}

}  // namespace

extern "C" {

int dsim_batch_create(uint64_t spinCapacity, uint32_t jobCapacity, dsim_batch** out) {
    if (!out || spinCapacity == 0 || jobCapacity == 0 || spinCapacity > 0xFFFFFFE0ull) {
        set_last_error(kErrInvalid, "dsim_batch_create: bad argument");
        return kErrInvalid;
    }
    *out = nullptr;
    dsim_batch* b = new dsim_batch();
    b->cap = (spinCapacity + 31) & ~31ull;
    b->jobCap = jobCapacity;
    int rc = kOk;
    if (cudaStreamCreateWithFlags(&b->st, cudaStreamNonBlocking) != cudaSuccess) rc = kErrCuda;
    for (int k = 0; k < dsim_batch::kSide && !rc; k++)
        if (cudaStreamCreateWithFlags(&b->side[k], cudaStreamNonBlocking) != cudaSuccess ||
            cudaEventCreateWithFlags(&b->joinEv[k], cudaEventDisableTiming) != cudaSuccess)
            rc = kErrCuda;
    if (!rc && cudaEventCreateWithFlags(&b->forkEv, cudaEventDisableTiming) != cudaSuccess) rc = kErrCuda;
    for (int k = 0; k < 2 && !rc; k++) {
        for (int f = 0; f < kBF && !rc; f++) rc = balloc(b, (void**)&b->buf[k].f[f], b->cap * 4);
        for (int u = 0; u < kBU && !rc; u++) rc = balloc(b, (void**)&b->buf[k].u[u], b->cap * 4);
    }
    if (!rc) rc = balloc(b, (void**)&b->keys, b->cap * 4);
    if (!rc) rc = balloc(b, (void**)&b->d_jobs, (size_t)jobCapacity * sizeof(JobDev));
    if (!rc) rc = balloc(b, (void**)&b->d_subs, (size_t)b->subCap * sizeof(SubDev));
    if (!rc) rc = balloc(b, (void**)&b->d_counts, (size_t)4 * jobCapacity * 8);
    if (!rc) rc = balloc(b, (void**)&b->d_status, 4);
    if (!rc) rc = balloc(b, (void**)&b->d_stepNow, 4);
    if (!rc) rc = balloc(b, (void**)&b->d_trig, kTrig * sizeof(Trig));
    if (!rc && cudaMemcpy(b->d_trig, trig_table(), kTrig * sizeof(Trig), cudaMemcpyHostToDevice) != cudaSuccess) rc = kErrCuda;
    if (!rc && (cudaMemset(b->d_status, 0, 4) != cudaSuccess || cudaMemset(b->d_stepNow, 0, 4) != cudaSuccess ||
                cudaMemset(b->d_counts, 0, (size_t)4 * jobCapacity * 8) != cudaSuccess))
        rc = kErrCuda;
    if (rc) { dsim_batch_free(b); return rc; }
    *out = b;
    return kOk;
}

void dsim_batch_free(dsim_batch* b) {
    if (!b) return;
    if (b->st) cudaStreamSynchronize(b->st);
    invalidate_graph(b);
    for (int k = 0; k < 2; k++) {
        for (int f = 0; f < kBF; f++) cudaFree(b->buf[k].f[f]);
        for (int u = 0; u < kBU; u++) cudaFree(b->buf[k].u[u]);
        for (int f = 0; f < kBD; f++) cudaFree(b->buf[k].d[f]);
    }
    for (auto& j : b->jobs) cudaFree(j.wave);
    cudaFree(b->keys); cudaFree(b->hist); cudaFree(b->hstart); cudaFree(b->scratch);
    cudaFree(b->d_jobs); cudaFree(b->d_warps); cudaFree(b->d_subs); cudaFree(b->d_counts); cudaFree(b->d_status);
    cudaFree(b->d_stepNow); cudaFree(b->d_trig); cudaFree(b->d_sig);
    if (b->st) cudaStreamDestroy(b->st);
    for (int k = 0; k < dsim_batch::kSide; k++) {
        if (b->side[k]) cudaStreamDestroy(b->side[k]);
        if (b->joinEv[k]) cudaEventDestroy(b->joinEv[k]);
    }
    if (b->forkEv) cudaEventDestroy(b->forkEv);
    for (const dsim_cyl* c : b->cylsHeld) cyl_hold(c, -1);
    delete b;
}

static int add_sub(dsim_batch* b, const SubDev& s, const dsim_mesh* m, uint32_t* id) {
    if (b->subs.size() >= b->subCap) { set_last_error(kErrTooLarge, "batch: too many substrates"); return kErrTooLarge; }
    b->subs.push_back(s);
    b->meshes.push_back(m);
    DSIM_CUDA_TRY(cudaMemcpyAsync(b->d_subs + (b->subs.size() - 1), &s, sizeof(SubDev), cudaMemcpyHostToDevice, b->st));
    DSIM_CUDA_TRY(cudaStreamSynchronize(b->st));
    *id = (uint32_t)(b->subs.size() - 1);
    return kOk;
}

int dsim_batch_add_mesh(dsim_batch* b, const dsim_mesh* m, uint32_t* substrate) {
    if (!b || !m || !substrate) { set_last_error(kErrInvalid, "dsim_batch_add_mesh: null argument"); return kErrInvalid; }
    SubDev s;
    memset(&s, 0, sizeof(s));
    s.kind = kSubMesh;
    int rc = mesh_views(m, &s.g, &s.acc);
    if (rc) return rc;
    return add_sub(b, s, m, substrate);
}

int dsim_batch_add_cyl(dsim_batch* b, const dsim_cyl* c, uint32_t* substrate) {
    if (!b || !c || !substrate) { set_last_error(kErrInvalid, "dsim_batch_add_cyl: null argument"); return kErrInvalid; }
    SubDev s;
    memset(&s, 0, sizeof(s));
    s.kind = kSubCyl;
    int rc = cyl_view(c, &s.c);
    if (rc) return rc;
    if ((rc = add_sub(b, s, nullptr, substrate))) return rc;
    cyl_hold(c, 1);
    b->cylsHeld.push_back(c);
    return kOk;
}

// first precision-form job on a substrate: the mesh's FP64 triangle table, and
// for the batch the FP64 state fields of both spin buffers
static int ensure_precise(dsim_batch* b, uint32_t substrate) {
    int rc = kOk;
    SubDev& sd = b->subs[substrate];
    if (sd.kind == kSubMesh) {
        dsim_mesh* m = const_cast<dsim_mesh*>(b->meshes[substrate]);
        if ((rc = mesh_tri64(m))) return rc;
    }
    if (sd.kind == kSubMesh && !sd.g.tri64) {
        dsim_mesh* m = const_cast<dsim_mesh*>(b->meshes[substrate]);
        if ((rc = mesh_views(m, &sd.g, &sd.acc))) return rc;
        DSIM_CUDA_TRY(cudaMemcpyAsync(b->d_subs + substrate, &sd, sizeof(SubDev), cudaMemcpyHostToDevice, b->st));
        invalidate_graph(b);
    }
    if (!b->buf[0].d[0]) {
        for (int k = 0; k < 2; k++)
            for (int f = 0; f < kBD; f++)
                if ((rc = balloc(b, (void**)&b->buf[k].d[f], b->cap * 8))) return rc;
        invalidate_graph(b);
    }
    return kOk;
}

int dsim_batch_submit(dsim_batch* b, const dsim_job_desc* d, const float* pos3, const uint8_t* comp,
                      const uint32_t* fiber, uint32_t* jobId) {
    if (!b || !d || !pos3 || !comp || !jobId || d->nSpins == 0 || d->steps == 0 || d->substrate >= b->subs.size() ||
        !(d->deltaTime > 0.0f) || (d->waveform == DSIM_WAVE_TABLE && !d->table) || d->waveform > DSIM_WAVE_TABLE) {
        set_last_error(kErrInvalid, "dsim_batch_submit: bad argument");
        return kErrInvalid;
    }
    const uint32_t pad = (d->nSpins + 31u) & ~31u;
    if (b->N + pad > b->cap || b->jobs.size() >= b->jobCap) {
        set_last_error(kErrNoMem, "dsim_batch_submit: batch full (%llu + %u spins of %llu, %zu jobs of %u)",
                       (unsigned long long)b->N, pad, (unsigned long long)b->cap, b->jobs.size(), b->jobCap);
        return kErrNoMem;
    }
    const bool cyl = b->subs[d->substrate].kind == kSubCyl;
    BatchJob j;
    j.id = b->nextId;
    j.nSpins = d->nSpins;
    j.pad = pad;
    j.pc = (double)d->phaseConstant;
    JobDev& J = j.d;
    memset(&J, 0, sizeof(J));
    J.sub = d->substrate;
    J.steps = d->steps;
    J.start = b->stepNow;
    J.sortBits = sort_bits(d->nSpins);
    J.sortRegion = cyl ? 1u : 0u;
    for (int k = 0; k < 4; k++) { J.sd[k] = d->stepSd[k]; J.T2[k] = d->T2[k]; }
    J.perm = d->permeability;
    J.dt = d->deltaTime;
    J.clampHi = 1.0f - d->spinRadius;
    J.clampLo = -1.0f + d->spinRadius;
    J.reflType = d->reflectionType;
    J.maxSub = 4096;
    J.inR = d->innerRadiusProportion * d->innerRadiusProportion;
    J.key0 = (uint32_t)d->seed;
    J.key1 = (uint32_t)(d->seed >> 32);
    J.flags = d->flags & (DSIM_JOB_PRECISE | DSIM_JOB_LOCAL);
    if (J.flags == (DSIM_JOB_PRECISE | DSIM_JOB_LOCAL)) {
        set_last_error(kErrInvalid, "dsim_batch_submit: DSIM_JOB_PRECISE and DSIM_JOB_LOCAL exclude each other");
        return kErrInvalid;
    }
    J.spinR = d->spinRadius;
    if (J.flags) {
        int rc = ensure_precise(b, d->substrate);
        if (rc) return rc;
    }
    std::vector<float> w = make_wave(d);
    int rc = balloc(b, (void**)&j.wave, w.size() * 4);
    if (rc) return rc;
    J.wave = j.wave;
    if (!J.wave || w.size() < J.steps) {
        cudaFree(j.wave);
        set_last_error(kErrInvalid, "dsim_batch_submit: waveform table missing");
        return kErrInvalid;
    }
    if (cudaMemcpyAsync(j.wave, w.data(), w.size() * 4, cudaMemcpyHostToDevice, b->st) != cudaSuccess) {
        cudaFree(j.wave);
        set_last_error(kErrCuda, "dsim_batch_submit: waveform upload");
        return kErrCuda;
    }
    // host staging of the packed slots [N, N + pad)
    std::vector<float> hf[kBF];
    std::vector<uint32_t> hu[kBU];
    for (int f = 0; f < kBF; f++) hf[f].assign(pad, 0.0f);
    for (int u = 0; u < kBU; u++) hu[u].assign(pad, 0u);
    const uint32_t jobIndex = (uint32_t)b->jobs.size();
    for (uint32_t k = 0; k < pad; k++) {
        hu[U_JOB][k] = jobIndex;
        if (k < d->nSpins) {
            hf[F_X][k] = pos3[3 * k]; hf[F_Y][k] = pos3[3 * k + 1]; hf[F_Z][k] = pos3[3 * k + 2];
            hf[F_MAG][k] = 1.0f;
            uint32_t fb = fiber ? fiber[k] : 0xFFFFFFFFu;
            fb = cyl ? (fb & 0xFFFFFFu) : (fb & 0xFFFFu);
            hu[U_META][k] = (uint32_t)comp[k] | (fb << 8);
            hu[U_ID][k] = k;
        } else {
            hu[U_ID][k] = 0xFFFFFFFFu;
        }
    }
    for (int f = 0; f < kBF; f++)
        DSIM_CUDA_TRY(cudaMemcpyAsync(b->buf[b->cur].f[f] + b->N, hf[f].data(), (size_t)pad * 4, cudaMemcpyHostToDevice, b->st));
    for (int u = 0; u < kBU; u++)
        DSIM_CUDA_TRY(cudaMemcpyAsync(b->buf[b->cur].u[u] + b->N, hu[u].data(), (size_t)pad * 4, cudaMemcpyHostToDevice, b->st));
    if (J.flags) {
        // the FP64 state of the precision and cell-local forms: the given positions, magnitude 1
        std::vector<double> hd[kBD];
        for (int f = 0; f < kBD; f++) hd[f].assign(pad, 0.0);
        for (uint32_t k = 0; k < d->nSpins; k++) {
            hd[D_X][k] = pos3[3 * k]; hd[D_Y][k] = pos3[3 * k + 1]; hd[D_Z][k] = pos3[3 * k + 2];
            hd[D_MAG][k] = 1.0;
        }
        for (int f = 0; f < kBD; f++)
            DSIM_CUDA_TRY(cudaMemcpyAsync(b->buf[b->cur].d[f] + b->N, hd[f].data(), (size_t)pad * 8, cudaMemcpyHostToDevice, b->st));
        DSIM_CUDA_TRY(cudaStreamSynchronize(b->st));
    }
    b->jobs.push_back(j);
    b->nextId++;
    b->N += pad;
    if ((rc = layout_keys(b)) || (rc = upload_jobs(b))) return rc;
    DSIM_CUDA_TRY(cudaMemsetAsync(b->d_counts + 4 * jobIndex, 0, 32, b->st));
    DSIM_CUDA_TRY(cudaStreamSynchronize(b->st));
    b->warpsValid = false;
    *jobId = j.id;
    return kOk;
}

int dsim_batch_configure(dsim_batch* b, uint32_t chunk, uint32_t occupancy, uint32_t graphChunks) {
    if (!b || chunk == 0 || (occupancy != 4 && occupancy != 5 && occupancy != 6 && occupancy != 8)) {
        set_last_error(kErrInvalid, "dsim_batch_configure: chunk > 0, occupancy 4, 5, 6 or 8");
        return kErrInvalid;
    }
    b->chunk = chunk;
    b->chunkSet = true;
    b->occupancy = occupancy;
    b->graphChunks = graphChunks;
    b->warpsValid = false;  // the warps go by them
    invalidate_graph(b);
    return kOk;
}

int dsim_batch_block(const dsim_batch* b, uint32_t* threads) {
    if (!b || !threads) return kErrInvalid;
    *threads = b->blockThreads;
    return kOk;
}

int dsim_batch_set_block(dsim_batch* b, uint32_t threads) {
    if (!b || (threads != 64 && threads != 128 && threads != 256)) {
        set_last_error(kErrInvalid, "dsim_batch_set_block: 64, 128 or 256 threads");
        return kErrInvalid;
    }
    b->blockThreads = threads;
    invalidate_graph(b);
    return kOk;
}

static uint32_t remaining_steps(const dsim_batch* b) {
    uint32_t r = 0;
    for (const auto& j : b->jobs) {
        if (j.retired || job_finished(b, j)) continue;
        uint32_t left = j.d.steps - (b->stepNow - j.d.start);
        r = std::max(r, left);
    }
    return r;
}

// Steps of the next launch when the caller left the chunk to the batch: up to
// kLongChunk (a sort and a launch cost as much as a few steps, and a launch's
// wait for its slowest warp is paid once), but not far past the end of a job,
// so that the others' warps are listed again without it.
static uint32_t long_chunk(const dsim_batch* b, uint32_t steps) {
    constexpr uint32_t kLongChunk = 1000, kShortest = 100;
    uint32_t n = std::min(steps, kLongChunk);
    for (const auto& j : b->jobs) {
        if (job_finished(b, j)) continue;
        const uint32_t left = j.d.steps - (b->stepNow - j.d.start);
        if (left >= kShortest && left < n) n = left;
    }
    n = std::max(n, std::min(steps, kShortest));
    return n;
}

int dsim_batch_advance(dsim_batch* b, uint32_t steps) {
    if (!b) return kErrInvalid;
    if (b->N == 0 || steps == 0) return kOk;
    uint32_t chunks = (steps + b->chunk - 1) / b->chunk;
    if (!b->chunkSet) {
        uint32_t left = chunks * b->chunk;  // whole default chunks, as documented
        while (left > 0) {
            int rc = ensure_warps(b);
            if (rc) return rc;
            const uint32_t n = long_chunk(b, left);
            if ((rc = enqueue_chunk(b, n))) return rc;
            b->stepNow += n;
            left -= n;
        }
        return kOk;
    }
    const uint32_t G = b->graphChunks & ~1u;
    while (chunks > 0) {
        int rc = ensure_warps(b);
        if (rc) return rc;
        if (G > 0 && chunks >= G) {
            if (!b->graphValid || b->graphCur != b->cur) {
                if ((rc = capture_graph(b))) return rc;
            }
            DSIM_CUDA_TRY(cudaGraphLaunch(b->exec, b->st));
            b->graphLaunches++;
            b->launches += chunk_launches(b) * G;
            b->stepNow += G * b->chunk;
            chunks -= G;
        } else {
            if ((rc = enqueue_chunk(b, b->chunk))) return rc;
            b->stepNow += b->chunk;
            chunks--;
        }
    }
    return kOk;
}

int dsim_batch_run(dsim_batch* b) {
    if (!b) return kErrInvalid;
    uint32_t left = remaining_steps(b);
    int rc = dsim_batch_advance(b, left);
    if (rc) return rc;
    DSIM_CUDA_TRY(cudaStreamSynchronize(b->st));
    return kOk;
}

int dsim_batch_job_status(dsim_batch* b, uint32_t jobId, uint32_t* stepsDone, int* done) {
    BatchJob* j = b ? find_job(b, jobId) : nullptr;
    if (!j) { set_last_error(kErrInvalid, "dsim_batch_job_status: unknown job %u", jobId); return kErrInvalid; }
    uint32_t s = b->stepNow >= j->d.start ? std::min(b->stepNow - j->d.start, j->d.steps) : 0u;
    if (stepsDone) *stepsDone = s;
    if (done) *done = s >= j->d.steps ? 1 : 0;
    return kOk;
}

int dsim_batch_signal(dsim_batch* b, uint32_t jobId, const float* gradScaled, uint32_t nG, double* out) {
    return dsim_batch_signal_region(b, jobId, gradScaled, nG, 0.0, out);
}

int dsim_batch_signal_region(dsim_batch* b, uint32_t jobId, const float* gradScaled, uint32_t nG, double region,
                             double* out) {
    BatchJob* j = b ? find_job(b, jobId) : nullptr;
    if (!j || !gradScaled || !out || nG == 0 || !(region >= 0.0)) {
        set_last_error(kErrInvalid, "dsim_batch_signal: bad argument");
        return kErrInvalid;
    }
    // warps: 32 gradients x one spin segment each, about 16 warps per SM in all,
    // segments of whole windows of 32 spins
    const uint32_t gw = (nG + 31u) / 32u;
    const uint32_t most = std::max<uint32_t>(1u, std::min<uint32_t>((j->pad + 63u) / 64u, std::max<uint32_t>(1u, 2432u / gw)));
    const uint32_t segLen = ((j->pad + most - 1u) / most + 31u) & ~31u;
    const uint32_t nseg = (j->pad + segLen - 1u) / segLen;
    // phase = phaseConstant * (g . M)
    std::vector<double> kg(3 * (size_t)nG);
    for (size_t k = 0; k < kg.size(); k++) kg[k] = j->pc * (double)gradScaled[k];
    const size_t np = (size_t)nseg * nG * 15, need = kg.size() + np + (size_t)nG * 15;
    if (need > b->sigCap) {
        cudaFree(b->d_sig);
        b->bytes -= b->sigCap * 8;
        b->d_sig = nullptr; b->sigCap = 0;
        int rc = balloc(b, (void**)&b->d_sig, need * 8);
        if (rc) return rc;
        b->sigCap = need;
    }
    double *dk = b->d_sig, *dp = dk + kg.size(), *dout = dp + np;
    cudaError_t e = cudaMemcpyAsync(dk, kg.data(), kg.size() * 8, cudaMemcpyHostToDevice, b->st);
    if (e == cudaSuccess) {
        const uint32_t warps = gw * nseg;
        k_batch_signal<<<(warps * 32u + kSigThreads - 1) / kSigThreads, kSigThreads, 0, b->st>>>(
            view(b, b->cur), (uint32_t)j->slot0, j->pad, dk, nG, gw, nseg, segLen, region,
            j->d.flags != 0 && b->buf[b->cur].d[0] != nullptr, b->d_trig, dp);
        k_batch_signal_final<<<(nG * 15 + 31) / 32, dim3(32, 16), 0, b->st>>>(dp, nseg, nG, dout);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(out, dout, (size_t)nG * 15 * 8, cudaMemcpyDeviceToHost, b->st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(b->st);
    if (e != cudaSuccess) { set_last_cuda_error(e, "dsim_batch_signal", __FILE__, __LINE__); return kErrCuda; }
    return kOk;
}

int dsim_batch_get(dsim_batch* b, uint32_t jobId, float* pos3, float* mag, float* moments6, uint8_t* compartment,
                   uint32_t* fiber) {
    BatchJob* j = b ? find_job(b, jobId) : nullptr;
    if (!j) { set_last_error(kErrInvalid, "dsim_batch_get: unknown job %u", jobId); return kErrInvalid; }
    const uint32_t n = j->nSpins;
    float *dp = nullptr, *dm = nullptr, *dmo = nullptr;
    uint32_t* dme = nullptr;
    int rc;
    if ((rc = balloc(b, (void**)&dp, (size_t)n * 12)) || (rc = balloc(b, (void**)&dm, (size_t)n * 4)) ||
        (rc = balloc(b, (void**)&dmo, (size_t)n * 24)) || (rc = balloc(b, (void**)&dme, (size_t)n * 4))) {
        cudaFree(dp); cudaFree(dm); cudaFree(dmo); cudaFree(dme);
        return rc;
    }
    b->bytes -= (size_t)n * 44;
    k_batch_gather<<<(j->pad + 255) / 256, 256, 0, b->st>>>(view(b, b->cur), (uint32_t)j->slot0, j->pad, dp, dm, dmo, dme);
    cudaError_t e = cudaGetLastError();
    std::vector<float> hp(3 * (size_t)n), hm(n), hmo(6 * (size_t)n);
    std::vector<uint32_t> hme(n);
    if (e == cudaSuccess) e = cudaMemcpyAsync(hp.data(), dp, (size_t)n * 12, cudaMemcpyDeviceToHost, b->st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(hm.data(), dm, (size_t)n * 4, cudaMemcpyDeviceToHost, b->st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(hmo.data(), dmo, (size_t)n * 24, cudaMemcpyDeviceToHost, b->st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(hme.data(), dme, (size_t)n * 4, cudaMemcpyDeviceToHost, b->st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(b->st);
    cudaFree(dp); cudaFree(dm); cudaFree(dmo); cudaFree(dme);
    if (e != cudaSuccess) { set_last_cuda_error(e, "dsim_batch_get", __FILE__, __LINE__); return kErrCuda; }
    if (pos3) memcpy(pos3, hp.data(), hp.size() * 4);
    if (mag) memcpy(mag, hm.data(), hm.size() * 4);
    if (moments6) memcpy(moments6, hmo.data(), hmo.size() * 4);
    for (uint32_t k = 0; k < n; k++) {
        if (compartment) compartment[k] = (uint8_t)(hme[k] & 0xFFu);
        if (fiber) fiber[k] = hme[k] >> 8;
    }
    return kOk;
}

int dsim_batch_get_precise(dsim_batch* b, uint32_t jobId, double* pos3, double* mag) {
    BatchJob* j = b ? find_job(b, jobId) : nullptr;
    if (!j || !j->d.flags) {
        set_last_error(kErrInvalid, "dsim_batch_get_precise: %u is neither a precision-form nor a cell-local job", jobId);
        return kErrInvalid;
    }
    const uint32_t n = j->nSpins;
    double *dp = nullptr, *dm = nullptr;
    int rc;
    if ((rc = balloc(b, (void**)&dp, (size_t)n * 24)) || (rc = balloc(b, (void**)&dm, (size_t)n * 8))) {
        cudaFree(dp); cudaFree(dm);
        return rc;
    }
    b->bytes -= (size_t)n * 32;
    k_batch_gather64<<<(j->pad + 255) / 256, 256, 0, b->st>>>(view(b, b->cur), (uint32_t)j->slot0, j->pad, dp, dm);
    cudaError_t e = cudaGetLastError();
    std::vector<double> hp(3 * (size_t)n), hm(n);
    if (e == cudaSuccess) e = cudaMemcpyAsync(hp.data(), dp, (size_t)n * 24, cudaMemcpyDeviceToHost, b->st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(hm.data(), dm, (size_t)n * 8, cudaMemcpyDeviceToHost, b->st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(b->st);
    cudaFree(dp); cudaFree(dm);
    if (e != cudaSuccess) { set_last_cuda_error(e, "dsim_batch_get_precise", __FILE__, __LINE__); return kErrCuda; }
    if (pos3) memcpy(pos3, hp.data(), hp.size() * 8);
    if (mag) memcpy(mag, hm.data(), hm.size() * 8);
    return kOk;
}

int dsim_batch_counts(dsim_batch* b, uint32_t jobId, uint64_t counts[2]) {
    if (!b || !counts) return kErrInvalid;
    for (size_t k = 0; k < b->jobs.size(); k++) {
        if (b->jobs[k].id != jobId) continue;
        unsigned long long c[4];
        DSIM_CUDA_TRY(cudaMemcpyAsync(c, b->d_counts + 4 * k, 32, cudaMemcpyDeviceToHost, b->st));
        DSIM_CUDA_TRY(cudaStreamSynchronize(b->st));
        counts[0] = c[0]; counts[1] = c[1];
        return kOk;
    }
    set_last_error(kErrInvalid, "dsim_batch_counts: unknown job %u", jobId);
    return kErrInvalid;
}

int dsim_batch_precision_counts(dsim_batch* b, uint32_t jobId, uint64_t out[2]) {
    if (!b || !out) return kErrInvalid;
    for (size_t k = 0; k < b->jobs.size(); k++) {
        if (b->jobs[k].id != jobId) continue;
        unsigned long long c[4];
        DSIM_CUDA_TRY(cudaMemcpyAsync(c, b->d_counts + 4 * k, 32, cudaMemcpyDeviceToHost, b->st));
        DSIM_CUDA_TRY(cudaStreamSynchronize(b->st));
        out[0] = c[2]; out[1] = c[3];
        return kOk;
    }
    set_last_error(kErrInvalid, "dsim_batch_precision_counts: unknown job %u", jobId);
    return kErrInvalid;
}

uint32_t dsim_batch_status(dsim_batch* b) {
    if (!b) return 0;
    uint32_t s = 0;
    if (cudaMemcpyAsync(&s, b->d_status, 4, cudaMemcpyDeviceToHost, b->st) != cudaSuccess ||
        cudaStreamSynchronize(b->st) != cudaSuccess)
        return 0xFFFFFFFFu;
    return s;
}

int dsim_batch_retire(dsim_batch* b, uint32_t jobId) {
    BatchJob* j = b ? find_job(b, jobId) : nullptr;
    if (!j) { set_last_error(kErrInvalid, "dsim_batch_retire: unknown job %u", jobId); return kErrInvalid; }
    j->retired = true;
    return kOk;
}

int dsim_batch_compact(dsim_batch* b) {
    if (!b) return kErrInvalid;
    bool any = false;
    for (auto& j : b->jobs) any |= j.retired;
    if (!any) return kOk;
    const size_t nj = b->jobs.size();
    std::vector<int32_t> map(nj, -1);
    std::vector<int64_t> shift(nj, 0);
    std::vector<BatchJob> kept;
    std::vector<unsigned long long> oldCounts(4 * nj), newCounts;
    if (nj) {
        DSIM_CUDA_TRY(cudaMemcpyAsync(oldCounts.data(), b->d_counts, 32 * nj, cudaMemcpyDeviceToHost, b->st));
        DSIM_CUDA_TRY(cudaStreamSynchronize(b->st));
    }
    uint64_t slot = 0;
    for (size_t k = 0; k < nj; k++) {
        BatchJob& j = b->jobs[k];
        if (j.retired) { cudaFree(j.wave); j.wave = nullptr; continue; }
        map[k] = (int32_t)kept.size();
        shift[k] = (int64_t)slot - (int64_t)j.slot0;
        slot += j.pad;
        kept.push_back(j);
        for (int q = 0; q < 4; q++) newCounts.push_back(oldCounts[4 * k + q]);
    }
    int32_t* dmap = nullptr;
    int64_t* dshift = nullptr;
    int rc;
    if ((rc = balloc(b, (void**)&dmap, nj * 4)) || (rc = balloc(b, (void**)&dshift, nj * 8))) {
        cudaFree(dmap); cudaFree(dshift);
        return rc;
    }
    b->bytes -= nj * 12;
    cudaError_t e = cudaMemcpyAsync(dmap, map.data(), nj * 4, cudaMemcpyHostToDevice, b->st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(dshift, shift.data(), nj * 8, cudaMemcpyHostToDevice, b->st);
    if (e == cudaSuccess && b->N) {
        k_batch_compact<<<(uint32_t)((b->N + 255) / 256), 256, 0, b->st>>>(view(b, b->cur), view(b, 1 - b->cur), dmap, dshift);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(b->st);
    cudaFree(dmap); cudaFree(dshift);
    if (e != cudaSuccess) { set_last_cuda_error(e, "dsim_batch_compact", __FILE__, __LINE__); return kErrCuda; }
    b->cur = 1 - b->cur;
    b->jobs = kept;
    b->N = slot;
    b->warpsValid = false;
    if ((rc = layout_keys(b)) || (rc = upload_jobs(b))) return rc;
    if (!newCounts.empty())
        DSIM_CUDA_TRY(cudaMemcpyAsync(b->d_counts, newCounts.data(), newCounts.size() * 8, cudaMemcpyHostToDevice, b->st));
    DSIM_CUDA_TRY(cudaStreamSynchronize(b->st));
    invalidate_graph(b);
    return kOk;
}

// Autotuner: times the same max(trialSteps, 1000) steps (a multiple of every
// candidate chunk) of the current jobs for each candidate (step-kernel
// occupancy x chunk length x fine-grid cells per reference cell edge of every
// mesh substrate) from a snapshot of the spin state, restores the snapshot and
// keeps the fastest configuration.
int dsim_batch_autotune(dsim_batch* b, uint32_t trialSteps, uint32_t best[3], float* bestMs) {
    if (!b || !best || trialSteps == 0) { set_last_error(kErrInvalid, "dsim_batch_autotune: bad argument"); return kErrInvalid; }
    if (b->N == 0) { set_last_error(kErrInvalid, "dsim_batch_autotune: no jobs"); return kErrInvalid; }
    const bool hasD = b->buf[0].d[0] != nullptr;
    const size_t words = (size_t)(kBF + kBU + (hasD ? 2 * kBD : 0)) * b->N;
    uint32_t* snap = nullptr;
    int rc = balloc(b, (void**)&snap, words * 4);
    if (rc) return rc;
    b->bytes -= words * 4;
    const size_t nj = b->jobs.size();
    std::vector<unsigned long long> counts0(4 * nj);
    auto save = [&](void) -> cudaError_t {
        cudaError_t e = cudaSuccess;
        for (int f = 0; f < kBF && e == cudaSuccess; f++)
            e = cudaMemcpyAsync(snap + (size_t)f * b->N, b->buf[b->cur].f[f], b->N * 4, cudaMemcpyDeviceToDevice, b->st);
        for (int u = 0; u < kBU && e == cudaSuccess; u++)
            e = cudaMemcpyAsync(snap + (size_t)(kBF + u) * b->N, b->buf[b->cur].u[u], b->N * 4, cudaMemcpyDeviceToDevice, b->st);
        for (int f = 0; hasD && f < kBD && e == cudaSuccess; f++)
            e = cudaMemcpyAsync(snap + (size_t)(kBF + kBU + 2 * f) * b->N, b->buf[b->cur].d[f], b->N * 8,
                                cudaMemcpyDeviceToDevice, b->st);
        if (e == cudaSuccess) e = cudaMemcpyAsync(counts0.data(), b->d_counts, 32 * nj, cudaMemcpyDeviceToHost, b->st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(b->st);
        return e;
    };
    const int cur0 = b->cur;
    const uint32_t step0 = b->stepNow;
    auto restore = [&](void) -> cudaError_t {
        b->cur = cur0;
        cudaError_t e = cudaSuccess;
        for (int f = 0; f < kBF && e == cudaSuccess; f++)
            e = cudaMemcpyAsync(b->buf[b->cur].f[f], snap + (size_t)f * b->N, b->N * 4, cudaMemcpyDeviceToDevice, b->st);
        for (int u = 0; u < kBU && e == cudaSuccess; u++)
            e = cudaMemcpyAsync(b->buf[b->cur].u[u], snap + (size_t)(kBF + u) * b->N, b->N * 4, cudaMemcpyDeviceToDevice, b->st);
        for (int f = 0; hasD && f < kBD && e == cudaSuccess; f++)
            e = cudaMemcpyAsync(b->buf[b->cur].d[f], snap + (size_t)(kBF + kBU + 2 * f) * b->N, b->N * 8,
                                cudaMemcpyDeviceToDevice, b->st);
        b->stepNow = step0;
        b->warpsValid = false;  // jobs that finished in the trial run again
        if (e == cudaSuccess) e = cudaMemcpyAsync(b->d_stepNow, &b->stepNow, 4, cudaMemcpyHostToDevice, b->st);
        if (e == cudaSuccess) e = cudaMemcpyAsync(b->d_counts, counts0.data(), 32 * nj, cudaMemcpyHostToDevice, b->st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(b->st);
        return e;
    };
    // fine-grid resolutions: cells per reference-cell edge x 2
    const uint32_t gridHalves[] = {2, 3, 4, 5};  // 1, 1.5, 2, 2.5 fine cells per reference cell
    const uint32_t occs[] = {4, 5, 6, 8};
    const uint32_t chunks[] = {20, 40, 100, 200, 500, 1000};
    // the same steps for every candidate (a multiple of every chunk)
    const uint32_t T = std::max<uint32_t>((trialSteps + 999u) / 1000u * 1000u, 1000u);
    bool haveMesh = false;
    for (auto* m : b->meshes) haveMesh |= (m != nullptr);
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    float bestT = 3.4e38f;
    uint32_t bg = 0, bo = b->occupancy, bc = b->chunk;
    const uint32_t graph0 = b->graphChunks;
    const bool set0 = b->chunkSet;
    b->chunkSet = true;  // the candidates' chunks, and then the best one
    cudaError_t e = save();
    auto set_grid = [&](uint32_t halves) -> int {
        for (size_t k = 0; k < b->meshes.size(); k++) {
            if (!b->meshes[k]) continue;
            SubDev& sd = b->subs[k];
            uint32_t nf = std::min<uint32_t>(1024u, (sd.g.n * halves + 1) / 2);
            int r = mesh_rebuild_accel(const_cast<dsim_mesh*>(b->meshes[k]), nf);
            if (r) return r;
            r = mesh_views(b->meshes[k], &sd.g, &sd.acc);
            if (r) return r;
            if (cudaMemcpy(b->d_subs + k, &sd, sizeof(SubDev), cudaMemcpyHostToDevice) != cudaSuccess) return kErrCuda;
        }
        return kOk;
    };
    for (uint32_t gi = 0; gi < (haveMesh ? 4u : 1u) && e == cudaSuccess && !rc; gi++) {
        if (haveMesh && (rc = set_grid(gridHalves[gi]))) break;
        for (uint32_t oc : occs) {
            for (uint32_t ch : chunks) {
                if ((e = restore()) != cudaSuccess) break;
                b->occupancy = oc; b->chunk = ch; b->graphChunks = 0;
                invalidate_graph(b);
                cudaEventRecord(e0, b->st);
                if ((rc = dsim_batch_advance(b, T))) break;
                cudaEventRecord(e1, b->st);
                if ((e = cudaEventSynchronize(e1)) != cudaSuccess) break;
                float ms = 0.0f;
                cudaEventElapsedTime(&ms, e0, e1);
                ms *= (float)trialSteps / (float)T;  // per trialSteps steps
                if (ms < bestT) { bestT = ms; bg = haveMesh ? gridHalves[gi] : 0; bo = oc; bc = ch; }
            }
            if (rc || e != cudaSuccess) break;
        }
    }
    if (!rc && e == cudaSuccess && haveMesh) rc = set_grid(bg);
    // then the block size of the plain step kernels at that configuration
    uint32_t bt = b->blockThreads;
    const uint32_t shapes[] = {64, 128, 256};
    float bestShape = 3.4e38f;
    for (uint32_t th : shapes) {
        if (rc || e != cudaSuccess) break;
        if ((e = restore()) != cudaSuccess) break;
        b->occupancy = bo; b->chunk = bc; b->graphChunks = 0; b->blockThreads = th;
        invalidate_graph(b);
        cudaEventRecord(e0, b->st);
        if ((rc = dsim_batch_advance(b, T))) break;
        cudaEventRecord(e1, b->st);
        if ((e = cudaEventSynchronize(e1)) != cudaSuccess) break;
        float ms = 0.0f;
        cudaEventElapsedTime(&ms, e0, e1);
        ms *= (float)trialSteps / (float)T;
        if (ms < bestShape) { bestShape = ms; bt = th; }
    }
    if (bestShape < bestT) bestT = bestShape;
    b->blockThreads = bt;
    if (!rc && e == cudaSuccess) e = restore();
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(snap);
    b->occupancy = bo; b->chunk = bc; b->graphChunks = graph0;
    b->warpsValid = false;
    invalidate_graph(b);
    if (rc || e != cudaSuccess) b->chunkSet = set0;
    if (rc) return rc;
    if (e != cudaSuccess) { set_last_cuda_error(e, "dsim_batch_autotune", __FILE__, __LINE__); return kErrCuda; }
    best[0] = bo; best[1] = bc; best[2] = bg;
    if (bestMs) *bestMs = bestT;
    return kOk;
}

int dsim_batch_info(dsim_batch* b, uint64_t info[6]) {
    if (!b || !info) return kErrInvalid;
    uint64_t running = 0;
    for (const auto& j : b->jobs) running += (!j.retired && !job_finished(b, j)) ? 1 : 0;
    info[0] = b->N; info[1] = b->jobs.size(); info[2] = running; info[3] = b->bytes;
    info[4] = b->launches; info[5] = b->graphLaunches;
    return kOk;
}

int dsim_batch_sync(dsim_batch* b) {
    if (!b) return kErrInvalid;
    DSIM_CUDA_TRY(cudaStreamSynchronize(b->st));
    return kOk;
}

}  // extern "C"
