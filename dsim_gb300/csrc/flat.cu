// flat.cu -- the mesh step with warp-flattened candidate lists (kernel
// variants 5-9; 8 is the default).
//
// Same semantics as the reference's collision loop
// (rfdougherty/dSim dSim3/src/spinKernelCpu.cpp:198-499): for one sub-segment
// the first cell of the reference grid (in its x-outer, z-inner traversal of
// the box between the start and end cells) whose list holds a hit gives the
// nearest hit in that list, lowest index on ties, the last-hit triangle
// excluded.  Candidates come from a finer grid whose lists hold each triangle
// in every fine cell it touches; a collision round works in two flat passes
// over the whole warp:
//
//   1. cells: the lanes' fine-cell boxes are concatenated by a warp prefix sum;
//      32 cells at a time, lane m looks up its cell's record, so 32 loads are in
//      flight at once, and keeps it if the owner's sub-segment may meet its slab;
//   2. records: a second prefix sum concatenates the kept cells' records; lane j
//      tests flat record j, j + 32, ... against the owner's sub-segment, read
//      from a per-warp segment table in shared memory.
//
// Hits are filed in the owner's slots and resolved by the owner: the only hit,
// or the first reference cell (in the reference's order) whose list holds one,
// the nearest there, the lowest index on ties; the exact reference-grid scan
// when the slots overflowed.  Lanes do not advance through the steps in
// lockstep: a lane whose step ends starts its next step in the next round, so
// one lane's chain of reflections does not idle the other 31.
#include "common.cuh"
#include "engine.h"
#include "mesh_common.cuh"

#include "flat_round.cuh"

namespace dsim {

// and what only this kernel keeps of a lane
struct WalkLane : LaneState {
    float phase[32];
    uint32_t id[32];
};

// QUEUE (32-byte records): records past the plane test are finished 32 at a
// time from a per-warp queue (flat_round_mode's Q); STAGE: each cell's records
// staged in shared memory by bulk (TMA) copies, double-buffered
// (flat_round_mode's P)
template <bool STATS, int MINB, int LAYOUT, bool QUEUE = false, bool STAGE = false>
__global__ void __launch_bounds__(kFlatThreads, MINB) k_mesh_step_flat(MeshDev g, AccelDev acc,
                                                                       MeshStepArgs a, SpinsSorted S,
                                                                       int rng) {
    __shared__ FlatWarp wh[kFlatWarps];
    __shared__ WalkLane wc[kFlatWarps];
    __shared__ FlatQueue wq[QUEUE ? kFlatWarps : 1];
    __shared__ FlatStage ws[STAGE ? kFlatWarps : 1];
    const uint32_t FULL = 0xFFFFFFFFu;
    const uint32_t lane = threadIdx.x & 31u;
    FlatWarp& H = wh[threadIdx.x >> 5];
    if (STAGE) {
        if (lane == 0) stage_init(&ws[threadIdx.x >> 5]);
        __syncwarp();
    }
    const uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, warps = (S.N + a.perWarp - 1) / a.perWarp;
    const uint32_t w0 = w & ~(kDealWarps - 1u), dealt = min(kDealWarps, warps - w0);  // the warps that share spins
    const uint32_t i = w0 * a.perWarp + lane * dealt + (w - w0);
    const bool valid = w < warps && lane < a.perWarp && i < S.N;
    // the position is o at the top of a step, the start of its current sub-segment within one
    float ox = 0.0f, oy = 0.0f, oz = 0.0f;
    WalkLane& C = wc[threadIdx.x >> 5];
    float &mag = C.mag[lane], &phase = C.phase[lane], &umax = C.umax[lane], &umin = C.umin[lane], &u = C.u[lane];
    uint32_t &comp = C.comp[lane], &fiber = C.fiber[lane], &id = C.id[lane], &nrefl = C.nrefl[lane],
             &nperm = C.nperm[lane], &status = C.status[lane], &it = C.it[lane], &sub = C.sub[lane];
    mag = phase = umin = 0.0f;
    umax = u = 1.0f;
    comp = fiber = id = nrefl = nperm = status = it = sub = 0;
    uint32_t ntested = 0;
    if (valid) {
        ox = S.x[i]; oy = S.y[i]; oz = S.z[i]; mag = S.mag[i]; phase = S.phase[i];
        uint32_t meta = S.meta[i];
        comp = meta & 0xFFu; fiber = meta >> 8;
        id = S.id[i];
    }
    uint32_t k0 = a.key0, k1 = a.key1;
    if (valid && rng == kRngPhiloxPerSpinKey) { k0 = a.spinKeys[2 * id]; k1 = a.spinKeys[2 * id + 1]; }
    // Each lane runs its own step counter: a lane whose step ends in a round
    // starts its next step in the following round, so the warp's rounds are
    // not held back by the lane with the longest reflection chain of a step.
    bool active = valid && a.iterations > 0;
    bool fresh = active;  // the lane starts step `it` at the top of the round
    float px = ox, py = oy, pz = oz;
    uint32_t excluded = 0xFFFFFFFFu;
    while (__any_sync(FULL, active)) {
        if (fresh) {
            Draw d;
            if (rng == kRngReplay) {
                float4 q = __ldg(a.draws + (size_t)it * S.N + id);
                d.nx = q.x; d.ny = q.y; d.nz = q.z; d.u = q.w;
            } else {
                d = philox_draw(a.spinBase + id, a.step0 + it, a.stream, k0, k1);
            }
            u = d.u;
            const float sd = a.sd[comp & 3u];
            px = ox + d.nx * sd; py = oy + d.ny * sd; pz = oz + d.nz * sd;
            // the reference's endPos equals the sub-segment target p at the top
            // of every collision round, so p doubles as endPos
            excluded = 0xFFFFFFFFu;
            umax = 1.0f; umin = 0.0f;
            sub = 0;
            if (STATS) {
                uint32_t sx = ref_coord(ox, g.L, g.n), sy = ref_coord(oy, g.L, g.n), sz = ref_coord(oz, g.L, g.n);
                uint32_t tx = ref_coord(px, g.L, g.n), ty = ref_coord(py, g.L, g.n), tz = ref_coord(pz, g.L, g.n);
                for (uint32_t cx = min(sx, tx); cx <= max(sx, tx); cx++)
                    for (uint32_t cy = min(sy, ty); cy <= max(sy, ty); cy++)
                        for (uint32_t cz = min(sz, tz); cz <= max(sz, tz); cz++) {
                            uint32_t c = g.n * g.n * cz + g.n * cy + cx;
                            ntested += __ldg(g.cell_start + c + 1) - __ldg(g.cell_start + c);
                        }
            }
            fresh = false;
        }
        const bool open = active;  // every active lane has a sub-segment to test
        {
            bool found;
            FastHit best;
            flat_round_mode<LAYOUT>(H, g, acc, lane, open, ox, oy, oz, px, py, pz, excluded, found, best,
                                    QUEUE ? &wq[threadIdx.x >> 5] : nullptr, STAGE ? &ws[threadIdx.x >> 5] : nullptr);
            if (open) {
                bool finish = !found;
                if (found) {
                    apply_hit(g, best, u, a.perm, a.reflType, umax, umin, ox, oy, oz, px, py, pz, comp, fiber,
                              excluded, nrefl, nperm);
                    if (++sub >= a.maxSub) {
                        status |= kStatusSubsegCap;
                        px = ox; py = oy; pz = oz;
                        finish = true;
                    }
                }
                if (finish) {
                    // end of step `it`: clamp, T2 decay, phase
                    float ex = px, ey = py, ez = pz;
                    if (ex > a.clampHi) ex = a.clampHi; else if (ex < a.clampLo) ex = a.clampLo;
                    if (ey > a.clampHi) ey = a.clampHi; else if (ey < a.clampLo) ey = a.clampLo;
                    if (ez > a.clampHi) ez = a.clampHi; else if (ez < a.clampLo) ez = a.clampLo;
                    ox = ex; oy = ey; oz = ez;
                    mag += -mag / a.T2[comp & 3u] * a.dt;
                    float gx = a.gx, gy = a.gy, gz = a.gz;
                    if (a.grad) { float4 G = __ldg(a.grad + it); gx = G.x; gy = G.y; gz = G.z; }
                    phase += (gx * ox + gy * oy + gz * oz) * a.pc;
                    if (++it >= a.iterations) active = false;
                    else fresh = true;
                }
            }
            __syncwarp();
            if (STAGE && ws[threadIdx.x >> 5].abort) {  // warp-uniform: a staging wait ran out
                if (valid) atomicOr(a.status, (uint32_t)kStatusStageTimeout);
                return;
            }
        }
    }
    if (!valid) return;
    S.x[i] = ox; S.y[i] = oy; S.z[i] = oz; S.mag[i] = mag; S.phase[i] = phase;
    S.meta[i] = (comp & 0xFFu) | (fiber << 8);
    if (a.counts) { a.counts[2 * id] += nrefl; a.counts[2 * id + 1] += nperm; }
    if (STATS && a.tested) a.tested[id] += ntested;
    if (status) atomicOr(a.status, status);
}

// Spins per warp: below 32 of them at most 24 warps per SM, where a warp then
// still holds 16, else 20.  us per step at 12 / 16 / 20 / 24 / 28 warps per SM: 4096
// spins on 25 tubes with myelin 4.35 / 4.15 / 4.11 / 4.13 / 5.31; 30,000 spins on
// 100 tubes 7.01 / 6.28 / 6.18 / 6.63 / 7.33; 45,000 8.51 / 7.96 / 7.51 / 7.57 /
// 8.27; 60,000 9.85 / 9.16 / 8.76 / 8.72 / 9.29; 80,000 10.5 / 10.4 / 10.1 / 9.8 /
// 10.6; 65,536 on 25 tubes with myelin 14.9 / 13.6 / 12.9 / 12.4 / 13.0.  32 spins a
// warp at 1000 spins 12.9, at 8192 14.0.
uint32_t mesh_spins_per_warp(uint32_t N) {
    return spins_per_warp(N, N >= 24u * 16u * kSmCount ? 24 : 20, false);
}

int launch_mesh_step_flat(const MeshDev& g, const AccelDev& acc, const MeshStepArgs& args,
                          const SpinsSorted& S, int rng, cudaStream_t st, int occupancy, bool queue, bool stage) {
    if (S.N == 0 || args.iterations == 0) return kOk;
    MeshStepArgs a = args;
    a.perWarp = mesh_spins_per_warp(S.N);
    const uint32_t warps = (S.N + a.perWarp - 1) / a.perWarp;
    dim3 block(kFlatThreads), grid((warps + kFlatWarps - 1) / kFlatWarps);
    // one instantiation per record layout keeps each kernel's registers to its own path
    if (a.tested) k_mesh_step_flat<true, 4, 0><<<grid, block, 0, st>>>(g, acc, a, S, rng);
    else if (acc.wide == 2) {
        if (occupancy >= 8) k_mesh_step_flat<false, 8, 2><<<grid, block, 0, st>>>(g, acc, a, S, rng);
        else if (occupancy >= 6) k_mesh_step_flat<false, 6, 2><<<grid, block, 0, st>>>(g, acc, a, S, rng);
        else k_mesh_step_flat<false, 4, 2><<<grid, block, 0, st>>>(g, acc, a, S, rng);
    } else if (acc.wide == 1 && stage) {
        k_mesh_step_flat<false, 6, 1, false, true><<<grid, block, 0, st>>>(g, acc, a, S, rng);
    } else if (acc.wide == 1 && queue) {
        // Blocks per SM: as few of 4 (118 registers) to 7 (72, 32 B of spills) as
        // reach the fewest waves.  us per step on 100 tubes at 4 / 5 / 6 / 7, the
        // rule's marked: 70,000 spins 10.5* / 10.5 / 11.1 / 11.9; 90,000 16.0 /
        // 11.2* / 11.8 / 12.7; 100,000 16.8 / 15.5 / 12.2* / 13.0; 125,000 17.4 /
        // 17.1 / 17.7 / 13.7*; 150,000 19.1* / 18.6 / 19.5 / 20.4; 220,000 26.6 /
        // 25.2 / 22.4* / 23.9; 400,000 46.6 / 40.6 / 38.8 / 37.0*; 600,000 66.2 /
        // 57.7 / 55.5 / 55.4*
        const uint32_t k = blocks_per_sm(grid.x, 4, 7);
        if (k == 4) k_mesh_step_flat<false, 4, 1, true><<<grid, block, 0, st>>>(g, acc, a, S, rng);
        else if (k == 5) k_mesh_step_flat<false, 5, 1, true><<<grid, block, 0, st>>>(g, acc, a, S, rng);
        else if (k == 6) k_mesh_step_flat<false, 6, 1, true><<<grid, block, 0, st>>>(g, acc, a, S, rng);
        else k_mesh_step_flat<false, 7, 1, true><<<grid, block, 0, st>>>(g, acc, a, S, rng);
    } else if (acc.wide == 1) {
        if (occupancy >= 8) k_mesh_step_flat<false, 8, 1><<<grid, block, 0, st>>>(g, acc, a, S, rng);
        else if (occupancy >= 6) k_mesh_step_flat<false, 6, 1><<<grid, block, 0, st>>>(g, acc, a, S, rng);
        else k_mesh_step_flat<false, 4, 1><<<grid, block, 0, st>>>(g, acc, a, S, rng);
    } else {
        if (occupancy >= 6) k_mesh_step_flat<false, 6, 0><<<grid, block, 0, st>>>(g, acc, a, S, rng);
        else k_mesh_step_flat<false, 4, 0><<<grid, block, 0, st>>>(g, acc, a, S, rng);
    }
    DSIM_CUDA_TRY(cudaGetLastError());
    return kOk;
}

}  // namespace dsim
