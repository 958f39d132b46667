// piston.cuh — the velocity laws of the wave makers, and the block that
// evaluates them once per step.
#pragma once

#include "kernels.cuh"

namespace rrsph {
namespace {

// Piston velocity of dynamic_boundaries (RRSPH_OMP/src/WaveMaker.cpp:34-82)
// for one set of wave-maker parameters.
__device__ inline double piston_law_vx(int nwm, double phase, double freq, double H, double k, double depth,
                                double time_start, double time) {
    const double delta = phase - freq * time_start;
    const double omega = freq;
    const double kd = k * depth;
    const double sh = sinh(kd), ch = cosh(kd);
    const double m1 = 2 * (sh * sh) / (sh * ch + kd);
    const double S0 = H / m1;
    double vx = 0.5 * S0 * omega * cos(omega * time + delta);
    if (nwm == 3) {
        const double e2_1 = (H * H) / (32 * depth);
        const double e2_2 = 3 * ch / (sh * sh * sh) - 2 / m1;
        vx += 2 * omega * (e2_1 + e2_2) * cos(2 * omega * time + 2 * delta);
    }
    return vx;
}

// The params' piston, or X'(t) of the Fourier piston X(t) = sum_k c_k
// sin(k omega t) when one is set.
__device__ inline double piston_vx(const DevParams& P, double time) {
    if (P.fourier_n > 0) {
        double vx = 0;
        for (int k = 1; k <= P.fourier_n; k++) {
            const double phi = k * P.fourier_omega * cos(k * P.fourier_omega * time);
            vx += P.fourier_coef[k - 1] * phi;
        }
        return vx;
    }
    return piston_law_vx(P.nwm, P.nwm_phase, P.nwm_freq, P.nwm_H, P.nwm_k, P.depth, P.nwm_time_start, time);
}

// Piston velocity of nwm_solitary_rayleigh (WaveMaker.cpp:84-134).
__device__ inline double solitary_vx(const DevParams& P, double time) {
    const double H = P.nwm_H, h = P.depth, g = P.g;
    const double k = sqrt(3 * H / (4 * (h * h) * (H + h)));
    const double c = sqrt(g * (H + h));
    const double Tf = 2 / (k * c) * (3.8 + H / h);
    const double tau = k * c * (time - Tf);
    const double u = tanh(tau);
    const double top = k * H * (h + H - H * (u * u)) + 2 * k * ((H * u) * (H * u));
    const double b = k * (h + H - H * (u * u));
    const double dxdu = top / (b * b);
    const double th = tanh(tau);
    return dxdu * (1 - th * th) * (k * c);
}

__device__ __forceinline__ double params_vx(const DevParams& P, double time) {
    return P.nwm == 5 ? solitary_vx(P, time) : piston_vx(P, time);
}
__device__ __forceinline__ double table_vx(const PistonLaw& L, double time) {
    return piston_law_vx(L.nwm, L.phase, L.freq, L.H, L.k, L.depth, L.time_start, time);
}

// The step's piston velocities, by one extra block of a kernel that runs before
// the whole step and leaves the SMs room: a chain of some 200 FP64 operations
// (hyperbolic functions), which each piston particle's thread would run through at
// the end of the step. 2.5k tank, mixed: 28.2 -> 24.6 us a step; 409k flume,
// FP64: whole step 29 -> 23 us. Not in the mixed step's thread-per-particle density
// gather, which it slowed more (46.2 -> 48.2 us on the flume) than it gave.
__device__ __noinline__ void piston_block(const DevParams& P, const State& S, StepScalars* __restrict__ scal) {
    const double time = scal->time;
    if (S.wave_tank) {
        for (uint32_t w = threadIdx.x; w < S.wave_count; w += blockDim.x) S.wave_vx[w] = table_vx(S.wave_law[w], time);
    } else if (threadIdx.x == 0) {
        scal->piston_vx = params_vx(P, time);
    }
}

}  // namespace

// Whether a step has pistons for piston_block.
inline bool has_pistons(const DevParams& P, const State& S) {
    return S.wave_tank != nullptr || (P.nwm_valid && (P.nwm == 2 || P.nwm == 3 || P.nwm == 5));
}

}  // namespace rrsph
