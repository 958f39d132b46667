// step_particle.cuh — the per-particle pieces of the time step that more than
// one kernel runs: the geometry test, the key pass, predict_half_step, the
// piston laws and the whole step of one particle. The whole-step kernel runs
// them over all particles; the fused force + whole-step gather of the mixed
// step with neighbour reuse runs them for the particle whose acceleration it
// has just summed.
#pragma once

#include "kernels.cuh"
#include "neighbour.cuh"
#include "piston.cuh"

namespace rrsph {
namespace {

// predict_half_step (RRSPH_OMP/src/PredictHalfStep.cpp:4-23) fused with the
// key pass of make_grid (RRSPH_OMP/src/GridFind.cpp:55-75). Also clears the
// cell-table entries of the previous grid (key_of) so that the table needs no
// max_cells-sized reset.
// Cell key of particle i at (x, y, z) (GridFind.cpp:55-75); also clears the
// previous grid's cell-table entry of i and records the new key.
// Strictly inside the geometry box (WholeStep.cpp:4-17, ConsistencyCheck.cpp:162-218),
// the double compares done on the ordered bit patterns (a NaN is outside).
template <int DIM>
__device__ __forceinline__ bool in_geometry(const DevParams& P, double x, double y, double z) {
    const long long ox = dorder(x), oy = dorder(y);
    bool in = ox < P.oxmax && ox > P.oxmin && oy < P.oymax && oy > P.oymin && !dnan(x) && !dnan(y);
    if (DIM == 3) {
        const long long oz = dorder(z);
        in = in && oz < P.ozmax && oz > P.ozmin && !dnan(z);
    }
    return in;
}

// Compile-time variants of the per-particle kernels. A switch that is off in
// a variant leaves no instructions behind: the FP64 pipe (one lane per clock
// per SM on this part) also issues the predicated-off double instructions of
// small if-converted branches.
enum : int { kVarCont = 1, kVarRare = 2, kVarMixed = 4 };  // continuity, XSPH or dynamic dt, FP32-mixed
// M: 0 = FP64 step, 1 = FP32-mixed step, 2 = decided at run time from the state's buffers.

// A particle that moved more than half the skin since the build asks for a
// rebuild (one atomic per warp).
__device__ __forceinline__ void reuse_check(const State& S, bool moved) {
    const unsigned am = __activemask();
    const unsigned who = __ballot_sync(am, moved);
    if (who && (threadIdx.x & 31) == (unsigned)(__ffs(am) - 1)) atomicOr(S.vl_rebuild, 1u);
}

// Neighbour reuse, in the key pass of particle i: the velocity (and with
// continuity density VD4) copies of the next step at slot k.
template <int DIM>
__device__ __forceinline__ void velocity_copies(const DevParams& P, const State& S, const Sorted& G, uint32_t i,
                                                uint32_t k) {
    float4 v;
    if (DIM == 3) {
        v = S.vpf4[i];
        v.w = 0.0f;
    } else {
        const float2 v2 = S.vpf2[i];
        v = make_float4(v2.x, v2.y, 0.0f, 0.0f);  // .zw (summation): the density pass writes them
    }
    if (G.VD4n) {
        v.w = d2f(S.rho_pred[i]);
        G.VD4n[k] = vd4_of<DIM>(S.vx[i], S.vy[i], DIM == 3 ? S.vz[i] : 0.0, S.rho[i] - P.rho0);
    }
    G.V4n[k] = v;
}
// kReuseCell: the same copies and test with the position as the offset (ox, oy)
// from the edge of its cell (cx, cy).
__device__ __forceinline__ void reuse_cell_pass(const DevParams& P, const State& S, const Sorted& G, uint32_t i,
                                                uint32_t cx, uint32_t cy, float ox, float oy) {
    const uint32_t b = S.bcxy[i];
    const float2 bo = S.boff[i];
    // offset from the edge of the cell the particle had at the build
    const float px = ox + (float)((int)cx - (int)(b & 0xFFFFu)) * P.mf.cell;
    const float py = oy + (float)((int)cy - (int)(b >> 16)) * P.mf.cell;
    const uint32_t k = S.slot[i];
    reinterpret_cast<float4*>(G.posn)[k] = make_float4(px, py, 0.0f, __int_as_float(S.itype[i]));
    velocity_copies<2>(P, S, G, i, k);
    const float dx = px - bo.x, dy = py - bo.y;
    reuse_check(S, !(dx * dx + dy * dy <= P.vl_half_skin2));
}

// Neighbour reuse, in the key pass of particle i at fixed-point position (x, y,
// z) in cell (cx, cy, cz): the next step's cell-order copies at the particle's slot of
// the last build (a step that rebuilds overwrites them in its new order), the position
// for the next build, and the test whether the particle has moved too far since the
// last: its separation in fixed point, which repeats every 32 cells, and its cell,
// which an upload may have changed by any number of them. With continuity density V4.w
// is rho_predict and VD4 = (v, rho - rho0), as the reorder writes them. A particle
// outside the grid is searched on a fresh grid each step.
template <int DIM>
__device__ __forceinline__ void reuse_pass(const DevParams& P, const State& S, const Sorted& G, uint32_t i,
                                           uint32_t x, uint32_t y, uint32_t z, uint32_t cx, uint32_t cy, uint32_t cz,
                                           bool far) {
    // within 16 cells of the cell at the build, where the separation is the only one
    auto near_cell = [](uint32_t c, uint32_t at_build) { return c - at_build + 16u <= 32u; };
    bool near;
    const uint32_t k = S.slot[i];
    const int32_t type = S.itype[i];
    far = far && type != P.type_non_existent;  // an absent one is nobody's neighbour wherever it lies
    G.posn[k] = Pos{(int)x, (int)y, (int)z, Pos::code_of(type, P.type_non_existent, far)};
    velocity_copies<DIM>(P, S, G, i, k);
    float d2;
    if (DIM == 3) {
        const int4 b = S.bfix4[i];
        S.fix4[i] = make_int4((int)x, (int)y, (int)z, 0);
        const float dx = (float)(int)(x - (uint32_t)b.x) * P.rf.u, dy = (float)(int)(y - (uint32_t)b.y) * P.rf.u,
                    dz = (float)(int)(z - (uint32_t)b.z) * P.rf.u;
        d2 = dx * dx + dy * dy + dz * dz;
        near = near_cell(cx, (uint32_t)b.w & 0x3FFu) && near_cell(cy, (uint32_t)b.w >> 10 & 0x3FFu) &&
               near_cell(cz, (uint32_t)b.w >> 20);
    } else {
        const int2 b = S.bfix2[i];
        S.fix2[i] = make_int2((int)x, (int)y);
        const uint32_t bc = S.bcxy[i];
        const float dx = (float)(int)(x - (uint32_t)b.x) * P.rf.u, dy = (float)(int)(y - (uint32_t)b.y) * P.rf.u;
        d2 = dx * dx + dy * dy;
        near = near_cell(cx, bc & 0xFFFFu) && near_cell(cy, bc >> 16);
    }
    if (far) *S.vl_far = 1u;
    reuse_check(S, far || !near || d2 > P.vl_half_skin2);
}

template <int DIM, int M>
__device__ __forceinline__ void key_pass(const DevParams& P, const State& S, const Sorted& G, uint32_t i, double x,
                                         double y, double z, uint32_t* __restrict__ flags) {
    constexpr uint32_t cmax = DIM == 3 ? 0x3FFu : 0xFFFFu;
    constexpr bool FIX = M != 0;
    const CellSplit sx = cell_split<FIX>(x, P.xmin, P.cell, P.inv_cell, P.mf.cell, cmax);
    const CellSplit sy = cell_split<FIX>(y, P.ymin, P.cell, P.inv_cell, P.mf.cell, cmax);
    bool outside = sx.below || sy.below;
    uint64_t key;
    CellSplit sz{};
    if (DIM == 3) {
        sz = cell_split<FIX>(z, P.zmin, P.cell, P.inv_cell, P.mf.cell, cmax);
        outside = outside || sz.below;
        key = split3(sx.c) | (split3(sy.c) << 1) | (split3(sz.c) << 2);
    } else {
        key = split2(sx.c) | (split2(sy.c) << 1);
    }
    if (key >= P.max_cells || outside) {
        // cell_idx >= max_cells (GridFind.cpp:61-72); keep kernels in bounds
        if (P.consistency_check || key >= P.max_cells) atomicOr(flags, RRSPH_FLAG_OUT_OF_DOMAIN);
        if (key >= P.max_cells) key = P.max_cells - 1;
    }
    const uint32_t old = S.key_of[i];
    if (old < P.max_cells && !P.keep_cells) G.cell_start[old] = kEmpty;
    S.key_of[i] = (uint32_t)key;
    G.keys_in[i] = (uint32_t)key;
    G.ids_in[i] = i;
    if (M != 0 && P.reuse == kReuseFixed)
        reuse_pass<DIM>(P, S, G, i, sx.fix, sy.fix, sz.fix, (uint32_t)sx.c & cmax, (uint32_t)sy.c & cmax,
                        (uint32_t)sz.c & cmax, sx.far || sy.far || (DIM == 3 && sz.far));
    if (M == 1 && P.reuse == kReuseFixed) return;  // the loop's next grid is the reuse step's
    if (M == 0 && !(DIM == 3 ? (void*)S.coff4 : (void*)S.coff2)) return;
    // offsets from the edge of the cell the key names: the Morton code keeps 16
    // bits per axis in 2D and 10 in 3D (GridUtils.h:50-64, 92-104). A cell
    // coordinate whose key lies in the grid fits in 32 bits, so the dropped bits
    // convert from 32 bits (a 64-bit integer conversion would take the FP64 pipe);
    // beyond that the key is out of the domain and the step fails.
    if (DIM == 2 && (M == 1 || S.coff2)) {
        const float ox = sx.off + (float)(uint32_t)(sx.c & ~0xFFFFull) * P.mf.cell;
        const float oy = sy.off + (float)(uint32_t)(sy.c & ~0xFFFFull) * P.mf.cell;
        S.coff2[i] = make_float2(ox, oy);
        if (M != 0 && P.reuse == kReuseCell)
            reuse_cell_pass(P, S, G, i, (uint32_t)(sx.c & 0xFFFFu), (uint32_t)(sy.c & 0xFFFFu), ox, oy);
    } else if (DIM == 3 && (M == 1 || S.coff4)) {
        const float ox = sx.off + (float)(uint32_t)(sx.c & ~0x3FFull) * P.mf.cell;
        const float oy = sy.off + (float)(uint32_t)(sy.c & ~0x3FFull) * P.mf.cell;
        const float oz = sz.off + (float)(uint32_t)(sz.c & ~0x3FFull) * P.mf.cell;
        S.coff4[i] = make_float4(ox, oy, oz, 0.0f);
    }
}

// predict_half_step (PredictHalfStep.cpp:4-23) of particle i with time step
// dt; the mixed step keeps v_predict in float only.
template <int DIM, int M, bool CONT>
__device__ __forceinline__ void predict(const DevParams& P, const State& S, uint32_t i, double vx, double vy,
                                        double vz, double rho, double dt, double ax, double ay, double az) {
    const bool mixed = M == 1 || (M == 2 && (DIM == 2 ? S.vpf2 != nullptr : S.vpf4 != nullptr));
    if (M != 0 && mixed) {  // v* = v + a dt/2 in float: the forces read it in float
        const float hf = d2f(dhalf(dt));
        if (DIM == 2) {
            S.vpf2[i] = make_float2(fmaf(d2f(ax), hf, d2f(vx)), fmaf(d2f(ay), hf, d2f(vy)));
        } else {
            S.vpf4[i] = make_float4(fmaf(d2f(ax), hf, d2f(vx)), fmaf(d2f(ay), hf, d2f(vy)),
                                    fmaf(d2f(az), hf, d2f(vz)), 0.0f);
        }
    } else if (M != 1) {  // the reference's v + (a dt) * 0.5
        S.vpx[i] = vx + __dmul_rn(ax, dt) * 0.5;
        S.vpy[i] = vy + __dmul_rn(ay, dt) * 0.5;
        if (DIM == 3) S.vpz[i] = vz + __dmul_rn(az, dt) * 0.5;
    }
    if (CONT) S.rho_pred[i] = rho + __dmul_rn(S.drho[i], dt) * 0.5;
}


// dt of the step: scal->dt, or update_dt (UpdateAcceleration.cpp:15-29) under
// DT_CORRECTION_DYNAMIC (with the step's maxima when dt_reduce is set). One
// thread (first) reports a never-ending dt.
template <bool RARE>
__device__ __forceinline__ double step_dt(const DevParams& P, const StepScalars* __restrict__ scal,
                                          uint32_t* __restrict__ flags, bool first) {
    double dt = scal->dt;
    if (RARE && P.dt_method == 2) {
        const double amax = P.dt_reduce ? __longlong_as_double((long long)scal->amax_bits) : 0.0;
        const double mumax = P.dt_reduce ? __longlong_as_double((long long)scal->mumax_bits) : 0.0;
        const double min_dt_a = sqrt(P.h / amax);
        const double min_dt_mu = P.h / (P.c_eos + mumax);
        dt = P.cfl * fmin(min_dt_a, min_dt_mu);
        if (dt <= P.never_ending_dt && first) atomicOr(flags, RRSPH_FLAG_NEVER_ENDING);
    }
    return dt;
}

// The next step's scalars (time += dt, step + 1, counters reset), by one thread.
__device__ __forceinline__ void advance_scalars(const DevParams& P, const StepScalars* __restrict__ scal,
                                                StepScalars* __restrict__ next, double dt) {
    const double time = scal->time;
    next->time = time + dt;
    next->dt = dt;
    next->step = scal->step + 1;
    next->amax_bits = 0;
    next->mumax_bits = 0;
    next->pairs = 0;
    next->nwm_off = scal->nwm_off || (P.nwm == 4 && time >= P.nwm_time_start) ? 1ull : 0ull;
    next->pairs_total = scal->pairs_total + scal->pairs;
}

// The per-particle part of k_whole: make_waves for particle i, whole_step,
// the boundary check and (next_keys) the next step's predictor + key pass,
// with the acceleration (ax, ay, az) of this step's force evaluation. pre: the
// piston velocities of the step are in scal and S.wave_vx (piston_block).
template <int DIM, int V>
__device__ __forceinline__ void whole_particle(const DevParams& P, const State& S, const Sorted& G, uint32_t i,
                                               double dt, const StepScalars* __restrict__ scal,
                                               uint32_t* __restrict__ flags, int next_keys, bool pre, double ax,
                                               double ay, double az) {
    constexpr bool CONT = (V & kVarCont) != 0, RARE = (V & kVarRare) != 0;
    constexpr int M = (V & kVarMixed) ? 1 : 0;
    const double time = scal->time;
    const unsigned long long nwm_off = scal->nwm_off;
    const bool waves = P.nwm && !nwm_off && dorder(time) >= dorder(P.nwm_time_start);
    if (S.wave_tank) {  // a table of pistons (one per tank of an ensemble)
        const int32_t w = S.wave_tank[i];
        if (w >= 0) {
            const PistonLaw L = S.wave_law[w];
            if (time >= L.time_start) {
                const double vx = pre ? S.wave_vx[w] : table_vx(L, time);
                S.rx[i] = S.rx[i] + vx * dt;
                S.vx[i] = vx;
            }
        }
    } else if (waves && P.nwm_valid && i >= P.nwm_start && i < P.nwm_end) {
        if (P.nwm == 2 || P.nwm == 3 || P.nwm == 5) {
            const double vx = pre ? scal->piston_vx : params_vx(P, time);
            S.rx[i] = S.rx[i] + vx * dt;
            S.vx[i] = vx;
        } else if (P.nwm == 4) {
            S.itype[i] = P.type_non_existent;
            atomicOr(S.itype_changed, 1u);
        }
    }
    const double v_dt = scal->step ? dt : dhalf(dt);
    double rho = 0.0;
    if (CONT) {
        rho = S.rho[i] + S.drho[i] * v_dt;
        S.rho[i] = rho;
    }
    double x = S.rx[i], y = S.ry[i], z = DIM == 3 ? S.rz[i] : 0.0;
    double vx = S.vx[i], vy = S.vy[i], vz = DIM == 3 ? S.vz[i] : 0.0;
    bool in = true, in_known = false;  // the geometry test of the final position, once
    if (S.itype[i] > 0) {
        vx = vx + ax * v_dt;
        vy = vy + ay * v_dt;
        if (DIM == 3) vz = vz + az * v_dt;
        if (RARE && P.avg_vel) {
            vx += S.avx[i];
            vy += S.avy[i];
            if (DIM == 3) vz += S.avz[i];
        }
        S.vx[i] = vx;
        S.vy[i] = vy;
        if (DIM == 3) S.vz[i] = vz;
        const double nx = x + vx * dt, ny = y + vy * dt, nz = DIM == 3 ? z + vz * dt : 0.0;
        bool move = true;
        if (P.consistency_treatment == 2 || P.consistency_check) {
            in = in_geometry<DIM>(P, nx, ny, nz);
            in_known = true;
            if (P.consistency_treatment == 2 && !in) {  // CONSISTENCY_FIX (WholeStep.cpp:47-54)
                move = false;
                in_known = false;
                S.itype[i] = P.type_non_existent;
                atomicOr(S.itype_changed, 1u);
            }
        }
        if (move) {
            x = nx; y = ny; z = nz;
            S.rx[i] = x;
            S.ry[i] = y;
            if (DIM == 3) S.rz[i] = z;
        }
    }
    if (P.consistency_check) {  // check_particles_are_within_boundaries (ConsistencyCheck.cpp:147-218)
        if (!in_known) in = in_geometry<DIM>(P, x, y, z);
        if (!in) atomicOr(flags, RRSPH_FLAG_OUTSIDE_GEOMETRY);
    }
    if (next_keys) {
        // the next step's predict_half_step and cell keys, from the state just written
        predict<DIM, M, CONT>(P, S, i, vx, vy, vz, rho, dt, ax, ay, az);
        key_pass<DIM, M>(P, S, G, i, x, y, z, flags);
    }
}

}  // namespace
}  // namespace rrsph
