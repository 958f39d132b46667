// kernels_pairs64.cu — the FP64 step's pair sums with each pair evaluated once.
//
// The FP64 pipe bounds this step: it takes 1.7 lanes per clock and SM where the
// FP32 and integer pipes take 128, whatever lanes of a warp are active, and an
// IEEE square root or division costs it 7.5 multiply-adds. So the pair terms,
// which are symmetric (the kernel value, the coefficient of r_i - r_j in the
// acceleration, the continuity rate), are evaluated for one of the two
// directions only, by warps with every lane busy, and stored for both
// particles; each particle then adds its own up in the search's order. The
// bookkeeping this takes (masks, ranks, stores, loads) runs on the idle pipes.
//
//   k_pair_masks   neighbours of a particle as a bit mask per stencil cell, the
//                  number of neighbours before each cell, their count
//   k_pair_terms   each pair once: kernel value and gradient (summation
//                  density); or the continuity rate and the acceleration
//   k_pair_density rho, p of a particle from its stored kernel values
//   k_pair_forces  each pair once: its acceleration (summation density)
//   k_pair_sum     accelerations (and drho) from the stored ones
//
// Against the directed gathers (kernels_fp64.cu; both sides of a pair, IEEE
// forms, 22 of 32 lanes): the 409k flume's density and forces 1.93 -> 0.46 ms
// (masks 59 us, terms 131, density 33, forces 174, sum 40), 385k particles in 3D
// 8.25 -> 2.0 ms a step (masks 314 us, terms 1287, sum 272), the 6k dam break 189
// -> 46 us (its sort, 30 us of the 189, then 15). The FP64 pipe is 74-80 % busy in
// the pair passes.
//
// A pair of particles k < i is evaluated by k's warp. Neighbour number s of a
// particle (its rank in the search's order: cells in stencil order, ids
// ascending) has its value in slot s of the particle's column, slot * n +
// particle; the other side's rank comes from its mask and count of the opposite
// cell. Neighbours past the slots, and those of cells with more particles than
// a mask has bits, are evaluated in place by both particles.
#include "pairs64.cuh"
#include "piston.cuh"

namespace rrsph {

namespace {

__device__ __forceinline__ void warp_sum_add(unsigned long long* dst, unsigned long long v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xFFFFFFFFu, v, o);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(dst, v);
}

// Neighbours of each particle (find_neighbours, GridFind.cpp:112-189): a block
// takes 32 consecutive particles, one warp per stencil cell, so the lanes of a
// warp read the same few cells in step. The float test on the cell-relative
// offsets decides outside the guard band around the cutoff, the reference's
// double test inside it and for particles outside their cell (clamped, or
// beyond the key's bits), whose x the reorder set to NaN (+inf: non-existent).
// near: the neighbours at up to one h, and some just beyond. Then the neighbours, and the owned ones,
// in the cells before this one (saturated: a number past the slots is not stored).
// Issue-bound: a dozen instructions per candidate. A group of lanes per
// particle instead, a cell a lane, ran at 14 (3D: 9) lanes of 32: 124 us on the
// 409k flume, 2.8 ms on 385k particles in 3D.
template <int DIM>
__global__ void __launch_bounds__(32 * Pm<DIM>::nc, DIM == 3 ? 2 : 7) k_pair_masks(DevParams P, State S, Sorted G,
                                                                                        StepScalars* scal) {
    if (blockIdx.x * 32u >= P.n) {  // the extra block
        piston_block(P, S, scal);
        return;
    }
    using M = Pm<DIM>;
    using T = typename M::T;
    __shared__ uint32_t counts[M::nc][32];
    const uint32_t lane = threadIdx.x & 31u;
    const int c = threadIdx.x >> 5;
    const uint32_t k = blockIdx.x * 32u + lane;
    const bool active = k < P.n;
    T mask = 0, near = 0;
    uint32_t first = 0;
    bool over = false;
    if (active) {
        const float4 pj = G.P4[k];
        uint32_t cell;
        bool wraps;
        // (a non-existent particle has none: its x is infinite)
        if (stencil_cell<DIM>(P, G.key[k], c, cell, wraps) && __float_as_int(pj.x) != 0x7F800000) {
            const uint32_t s = G.cell_start[cell], end = G.cell_end[cell];
            const uint32_t e = s != kEmpty ? end : s;
            first = s;
            // of two cells that meet by a wrapped coordinate only one sees the other: such
            // pairs are not stored
            over = e - s > (wraps ? 0u : M::bits);
            if (!over) {
                const MixedF& F = P.mf;
                // one h, and the error of the float test above it
                const float h2 = F.h * F.h * (1.0f + 2e-5f);
                const float3 sh = stencil_shift<DIM>(c);
                const float shx = sh.x * F.cell - pj.x, shy = sh.y * F.cell - pj.y;
                const float shz = DIM == 3 ? sh.z * F.cell - pj.z : 0.0f;
                // a word of bits at a time, the loads of a batch together (an index past the
                // cell's end loads its last particle; its bit is dropped); in 2D, with half
                // as many in a cell, batches of two: 59 us on the 409k flume, of four 62; in
                // 3D of four: 314 us on 385k, one candidate at a time into 64-bit words 436
                constexpr uint32_t B = DIM == 3 ? 4 : 2;
#pragma unroll 1
                for (uint32_t s0 = s; s0 < e; s0 += 32) {
                    const uint32_t len = min(e - s0, 32u);
                    uint32_t in = 0, below = 0, close = 0;  // below the guard band, or its end; at up to one h
#pragma unroll 1
                    for (uint32_t j = 0; j < len; j += B) {
                        float4 q[B];
#pragma unroll
                        for (uint32_t u = 0; u < B; u++) q[u] = G.P4[min(s0 + j + u, e - 1u)];
                        uint32_t a = 0, b = 0, o = 0;
#pragma unroll
                        for (uint32_t u = 0; u < B; u++) {
                            const float dx = q[u].x + shx, dy = q[u].y + shy, dz = DIM == 3 ? q[u].z + shz : 0.0f;
                            const float d2 = DIM == 3 ? dx * dx + dy * dy + dz * dz : dx * dx + dy * dy;
                            if (d2 < F.cut2_lo) a |= 1u << u;
                            if (!(d2 >= F.cut2_hi)) b |= 1u << u;
                            if (d2 < h2) o |= 1u << u;
                        }
                        in |= a << j;
                        below |= b << j;
                        close |= o << j;
                    }
                    const uint32_t valid = 0xFFFFFFFFu >> (32u - len);
                    in &= valid;
                    close &= valid;
                    for (uint32_t band = below & valid & ~in; band; band &= band - 1) {
                        const uint32_t bit = __ffs(band) - 1, i = s0 + bit;
                        const D3 a = row<DIM>(G.pr, i), b = row<DIM>(G.pr, k);
                        const double r2 = exact_dist2<DIM>(__dsub_rn(a.x, b.x), __dsub_rn(a.y, b.y),
                                                           DIM == 3 ? __dsub_rn(a.z, b.z) : 0.0);
                        if (r2 < P.cut2 && G.itype[i] != P.type_non_existent) {
                            in |= 1u << bit;
                            if (r2 <= P.h * P.h) close |= 1u << bit;
                        }
                    }
                    mask |= (T)in << ((s0 - s) & (M::bits - 1));
                    near |= (T)close << ((s0 - s) & (M::bits - 1));
                }
                if (c == M::nc / 2) mask &= ~((T)1 << (k - s));  // not itself
            }
        }
    }
    // at most 27 x 64 neighbours, and owned ones, in 12 bits each
    const uint32_t cnt = M::popc(mask);
    const uint32_t own = c == M::nc / 2 ? M::popc(mask & ~(((T)2 << ((k - first) & (M::bits - 1))) - 1))
                                        : (first > k ? cnt : 0u);
    counts[c][lane] = cnt | own << 12 | (over ? 0x80000000u : 0u);
    __syncthreads();
    if (!active) return;
    uint32_t before = 0;
    for (int b = 0; b < c; b++) before += counts[b][lane] & 0x7FFFFFFFu;
    const uint32_t own_before = before >> 12;
    before &= 0xFFFu;
    M::masks(G)[(size_t)c * P.n + k] = mask;
    M::nears(G)[(size_t)c * P.n + k] = near;
    G.pfirst[(size_t)c * P.n + k] = first;
    G.pbefore[(size_t)c * P.n + k] = (uint8_t)min(before, 255u);
    if (G.pown) G.pown[(size_t)c * P.n + k] = (uint8_t)min(own_before, 255u);
    if (c == M::nc - 1) {
        uint32_t word = 0;
        for (int b = 0; b < M::nc; b++) word |= (counts[b][lane] >> 31) << b;
        M::masks(G)[(size_t)M::nc * P.n + k] = (T)word;
        G.pcount[k] = before + cnt;
    }
}

// The viscous part in the IEEE forms of the directed gathers, for what the seeds do
// not take (infinite velocities and densities, densities that sum to zero).
__device__ __noinline__ double visc_ieee(double h, double alpha_c, double beta, double vr, double sep, double rhos) {
    const double mu = h * vr / sep;
    return (beta * mu - alpha_c) * mu / (0.5 * rhos);
}
// The viscous part of the coefficient (artificial_viscosity_part,
// ArtificialViscosity.h:29-65) added to pf: Pi_ij for an approaching pair, with
// one quotient for its two divisions. vr = (v_j - v_i).(r_j - r_i).
__device__ __forceinline__ double add_visc(const DevParams& P, double pf, double vr, double d2, double rhos) {
    if (!negative(vr)) return pf;
    const PairConst& C = P.pc;
    const double sep = d2 + C.etq_h2;
    const double x = sep * rhos;
    const double r = inverse_40(x);
    const double e = fma(-x, r, 1.0);
    const double u = vr * r;
    if (no_number(u)) return pf + visc_ieee(P.h, P.av_alpha * P.c_av, P.av_beta, vr, sep, rhos);
    const double w = fma(u, e, u);
    double f = C.av_c;  // -2 h alpha c; 2 h (beta mu - alpha c) with a bulk term
    if (C.bulk) f = fma(C.av_beta2h, C.h * rhos * w, f);
    return fma(f, w, pf);
}

// Lennard-Jones coefficient of a fluid particle's boundary neighbour
// (external_force_part, ExtForce.h:15-60). Few pairs: the IEEE forms, since the
// twelfth power multiplies their error.
__device__ __noinline__ double lj_coef(double rr0, double D, double d2) {
    const double dist = sqrt(d2);
    if (!(dist < rr0)) return 0.0;
    const double rn = rr0 / dist;
    const double rn2 = rn * rn, rn4 = rn2 * rn2, rn8 = rn4 * rn4;
    return D * (rn8 * rn4 - rn4) / d2;
}
// Coefficients of r_i - r_k in the accelerations of k and of i (they differ by
// the Lennard-Jones part, which only the fluid particle of the two feels).
template <int DIM>
__device__ __forceinline__ void force_coefs(const DevParams& P, const PairConst& C, double s, double d2,
                                            D3 d, D3 vk, D3 vi, double rhok, double rhoi, double prk, double pri,
                                            int32_t tk, int32_t ti, double& ck, double& ci) {
    double pf = prk + pri;
    if (C.visc) {
        const double vr = dot<DIM>({vi.x - vk.x, vi.y - vk.y, DIM == 3 ? vi.z - vk.z : 0.0}, d);
        pf = add_visc(P, pf, vr, d2, rhok + rhoi);
    }
    ck = ci = s * pf;
    if (lj_pair(P, tk, ti)) {
        const double fl = lj_coef(C.lj_rr0, C.lj_D, d2);
        if (tk > 0) ck -= fl;
        else ci -= fl;
    }
}

// density_con's terms of a pair (Density.h:63-114): the rate is the same for
// both sides, the delta-SPH part divides by the neighbour's density.
template <int DIM>
__device__ __forceinline__ void rate_terms(const DevParams& P, const PairConst& C, const Sorted& G, uint32_t k,
                                           uint32_t i, double s, double d2, D3 d, double& tk, double& ti) {
    const D3 a = row<DIM>(G.pd, k), b = row<DIM>(G.pd, i);
    tk = ti = dot<DIM>({b.x - a.x, b.y - a.y, DIM == 3 ? b.z - a.z : 0.0}, d) * s;
    if (P.density_treatment == 2) {
        const double2 qk = reinterpret_cast<const double2*>(G.pe)[k], qi = reinterpret_cast<const double2*>(G.pe)[i];
        const double f = C.dhc2 * (qi.x - qk.x) * s;  // -2 dhc m (rho_i - rho_k) s
        tk = fma(f, qi.y, tk);
        ti = fma(-f, qk.y, ti);
        // coincident particles: the reference's (diff.dwdr) / dist^2 is 0/0
        if ((__double_as_longlong(d2) << 1) == 0) tk = ti = __longlong_as_double(0x7FF8000000000000ll);
    }
}

// The stored terms of a neighbour, one record: 2D summation density (ax, ay);
// else (ax, ay, az, rate), a whole 32-byte sector, since one side's is a
// scattered store.
template <int DIM, bool CONT>
constexpr int kRec = DIM == 3 || CONT ? 4 : 2;
template <int DIM, bool CONT>
__device__ __forceinline__ void put_record(const Sorted& G, size_t at, D3 f, double rate) {
    double2* const p = reinterpret_cast<double2*>(G.pf + at * kRec<DIM, CONT>);
    if (kRec<DIM, CONT> == 2)
        p[0] = make_double2(f.x, f.y);
    else
        asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(f.x), "d"(f.y), "d"(f.z), "d"(rate)
                     : "memory");
}
// Both sides: the products are made once unless the coefficients differ.
template <int DIM, bool CONT>
__device__ __forceinline__ void put_forces(const Sorted& G, uint32_t cap, uint32_t rk, uint32_t ri, size_t ak,
                                           size_t ai, double ck, double ci, bool differ, D3 d, double tk, double ti) {
    D3 f{ck * d.x, ck * d.y, DIM == 3 ? ck * d.z : 0.0};
    if (rk < cap) put_record<DIM, CONT>(G, ak, f, tk);
    if (differ) f = {ci * d.x, ci * d.y, DIM == 3 ? ci * d.z : 0.0};
    if (ri < cap) put_record<DIM, CONT>(G, ai, {flip(f.x), flip(f.y), DIM == 3 ? flip(f.z) : 0.0}, ti);
}

// Each pair once. Summation density: m W into both columns, m s kept by the
// owner with the other side's rank. Continuity density: the rates and the
// accelerations into both columns (they wait for no sum).
// FP64 operations a pair: 2D summation 12 in the near branch of the kernel, 16
// in the far one; 3D continuity about 40.
template <int DIM, bool CONT>
__device__ __forceinline__ void pair_terms(const DevParams& P, const Sorted& G) {
    extern __shared__ uint2 pair_stack[];
    const PairConst& C = P.pc;
    const uint32_t cap = C.cap;
    const size_t n = P.n;
    walk_pairs<DIM, true, !CONT>(P, G, pair_stack, [&](const uint2 e, bool active, auto near) {
        constexpr bool NEAR = decltype(near)::value;
        if (!active) return;
        const Pair q = pair_of(e, warp_first());
        const uint32_t k = q.k, i = q.i, rk = q.rank;
        const uint32_t ri = rank_of<DIM>(P, G, i, q.c, q.bit);
        const size_t ak = rk * n + k, ai = ri * n + i;
        if (CONT) {
            D3 a, b, va, vb;
            double rhok, rhoi, prk, pri;
            force_rows<DIM>(G, k, a, va, rhok, prk);
            force_rows<DIM>(G, i, b, vb, rhoi, pri);
            const int32_t yk = G.itype[k], yi = G.itype[i];
            const D3 d{b.x - a.x, b.y - a.y, DIM == 3 ? b.z - a.z : 0.0};
            const double d2 = dot<DIM>(d, d);
            const Kern kk = cubic<NEAR, false>(C, d2);
            double tk, ti, ck, ci;
            rate_terms<DIM>(P, C, G, k, i, kk.s, d2, d, tk, ti);
            force_coefs<DIM>(P, C, kk.s, d2, d, va, vb, rhok, rhoi, prk, pri, yk, yi, ck, ci);
            put_forces<DIM, true>(G, cap, rk, ri, ak, ai, ck, ci, lj_pair(P, yk, yi), d, tk, ti);
        } else {
            const D3 a = row<DIM>(G.pr, k), b = row<DIM>(G.pr, i);
            const D3 d{b.x - a.x, b.y - a.y, DIM == 3 ? b.z - a.z : 0.0};
            const Kern kk = cubic<NEAR, true>(C, dot<DIM>(d, d));
            if (rk < cap) G.pw[ak] = kk.w;
            if (ri < cap) G.pw[ai] = kk.w;
            if (q.order < cap) {
                G.ps[q.order * n + k] = kk.s;
                G.prank[q.order * n + k] = (uint8_t)min(ri, 255u);
            }
        }
    });
}

template <int DIM, bool CONT>
__global__ void __launch_bounds__(kMaxGatherThreads) k_pair_terms(DevParams P, Sorted G) {
    pair_terms<DIM, CONT>(P, G);
}
// (at most 80 registers, for 25 single warps on an SM: 139k particles 845 us a step with
// the 90 it takes else, so 807)
template <>
__global__ void __launch_bounds__(kMaxGatherThreads, 3) k_pair_terms<3, true>(DevParams P, Sorted G) {
    pair_terms<3, true>(P, G);
}

// The accelerations, each pair once (summation density). A pair that recedes
// (no viscosity) is done after 10 FP64 operations in 2D; the others (and the
// wall pairs) go on to a second stack, and 32 of them at a time take the 12
// more: half the pairs, where one pass costs every warp both (20 a pair, 205 us
// on the 409k flume).
template <int DIM>
struct Approach {  // a warp's second stack
    uint2 e[kStack];
    double dx[kStack], dy[kStack], dz[DIM == 3 ? kStack : 1], vr[kStack];
};
// (at most 64 registers, for 32 blocks of one warp on an SM)
template <int DIM>
__global__ void __launch_bounds__(kMaxGatherThreads, 4) k_pair_forces(DevParams P, Sorted G) {
    extern __shared__ double2 pair_shared[];
    Approach<DIM>& A = reinterpret_cast<Approach<DIM>*>(pair_shared)[threadIdx.x >> 5];
    uint2* const stacks = reinterpret_cast<uint2*>(reinterpret_cast<Approach<DIM>*>(pair_shared) + (blockDim.x >> 5));
    const PairConst& C = P.pc;
    const uint32_t cap = C.cap, lane = threadIdx.x & 31u;
    const size_t n = P.n;
    uint32_t held = 0;
    auto second = [&](uint32_t at) {
        const Pair q = pair_of(A.e[at], warp_first());
        const uint32_t k = q.k, i = q.i, rk = q.rank;
        const D3 d{A.dx[at], A.dy[at], DIM == 3 ? A.dz[at] : 0.0};
        const double vr = A.vr[at];
        D3 a, va;
        double rhok, rhoi, prk, pri;
        force_rows<DIM>(G, k, a, va, rhok, prk);
        force_rows<DIM>(G, i, a, va, rhoi, pri);
        const int32_t tk = G.itype[k], ti = G.itype[i];
        const double d2 = dot<DIM>(d, d);
        double s;
        uint32_t ri;
        if (q.order < cap) {
            s = G.ps[q.order * n + k];
            ri = G.prank[q.order * n + k];
        } else {
            s = cubic_any(C, d2).s;
            ri = rank_of<DIM>(P, G, i, q.c, q.bit);
        }
        double pf = prk + pri;
        if (C.visc) pf = add_visc(P, pf, vr, d2, rhok + rhoi);
        double ck = s * pf, ci = ck;
        const bool lj = lj_pair(P, tk, ti);
        if (lj) {
            const double fl = lj_coef(C.lj_rr0, C.lj_D, d2);
            if (tk > 0) ck -= fl;
            else ci -= fl;
        }
        put_forces<DIM, false>(G, cap, rk, ri, rk * n + k, ri * n + i, ck, ci, lj, d, 0.0, 0.0);
    };
    walk_pairs<DIM, false, true>(P, G, stacks, [&](const uint2 e, bool active, auto) {
        bool go_on = false;
        D3 d{0.0, 0.0, 0.0};
        double vr = 0.0;
        if (active) {
            const Pair q = pair_of(e, warp_first());
            const uint32_t k = q.k, i = q.i, rk = q.rank;
            D3 a, b, va, vb;
            double rhok, rhoi, prk, pri;
            force_rows<DIM>(G, k, a, va, rhok, prk);
            force_rows<DIM>(G, i, b, vb, rhoi, pri);
            d = {b.x - a.x, b.y - a.y, DIM == 3 ? b.z - a.z : 0.0};
            go_on = q.order >= cap || lj_pair(P, G.itype[k], G.itype[i]);
            if (C.visc) {
                vr = dot<DIM>({vb.x - va.x, vb.y - va.y, DIM == 3 ? vb.z - va.z : 0.0}, d);
                go_on = go_on || negative(vr);
            }
            if (!go_on) {
                const size_t ao = q.order * n + k;
                const uint32_t ri = G.prank[ao];
                const double c = G.ps[ao] * (prk + pri);
                put_forces<DIM, false>(G, cap, rk, ri, rk * n + k, ri * n + i, c, c, false, d, 0.0, 0.0);
            }
        }
        const uint32_t who = __ballot_sync(0xFFFFFFFFu, go_on);
        if (go_on) {
            const uint32_t at = held + __popc(who & ((1u << lane) - 1u));
            A.e[at] = e;
            A.dx[at] = d.x;
            A.dy[at] = d.y;
            if (DIM == 3) A.dz[at] = d.z;
            A.vr[at] = vr;
        }
        held += __popc(who);
        __syncwarp();
        if (held >= 32) {
            held -= 32;
            second(held + lane);
            __syncwarp();
        }
    });
    if (lane < held) second(lane);
}

// density_sum + EOS (Density.h:25-61, EOS.cpp:31-34) from the stored values:
// streams 8 bytes per neighbour.
template <int DIM>
__global__ void __launch_bounds__(kMaxGatherThreads) k_pair_density(DevParams P, State S, Sorted G,
                                                                   StepScalars* __restrict__ scal,
                                                                   uint32_t* __restrict__ flags) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t cnt = 0;
    if (k < P.n) {
        const PairConst& C = P.pc;
        uint32_t over, slots;
        const bool more = stored_slots<DIM>(P, G, k, over, slots);
        double acc = C.w0;
        const double* const w = G.pw + k;
#pragma unroll 8
        for (uint32_t s = 0; s < slots; s++) acc += w[(size_t)s * P.n];
        cnt = slots;
        if (more && G.itype[k] != P.type_non_existent) {
            unstored_neighbours<DIM>(P, G, k, over, slots, [&](uint32_t, D3, double d2) {
                acc += cubic_any(C, d2).w;
                cnt++;
            });
        }
        if (cnt > P.max_nb - 1) atomicOr(flags, RRSPH_FLAG_NEIGHBOUR_OVERFLOW);
        const double p = eos_p(P, acc);
        const double x = acc * acc, r = inverse_40(x), u = p * r;
        const double pr2 = fma(u, fma(-x, r, 1.0), u);
        if (DIM == 3) {
            G.pr[(size_t)k * 4 + 3] = acc;
            G.pv[(size_t)k * 4 + 3] = pr2;
        } else {
            reinterpret_cast<double2*>(G.pq)[k] = make_double2(acc, pr2);
        }
        const uint32_t id = G.id[k];
        S.rho[id] = acc;
        S.p[id] = p;
    }
    warp_sum_add(&scal->pairs, cnt);
}

// update_acceleration's sums (UpdateAcceleration.cpp:33-125), and density_con's
// with continuity density, from the stored terms: one addition per component
// and a record of 16 or 32 bytes per neighbour, streamed.
template <int DIM, bool CONT>
__global__ void __launch_bounds__(kMaxGatherThreads) k_pair_sum(DevParams P, State S, Sorted G,
                                                               StepScalars* __restrict__ scal,
                                                               uint32_t* __restrict__ flags) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t cnt = 0;
    if (k < P.n) {
        const PairConst& C = P.pc;
        const size_t n = P.n;
        uint32_t over, slots;
        const bool more = stored_slots<DIM>(P, G, k, over, slots);
        double ax = 0.0, ay = -P.g, az = 0.0, rate = 0.0;
        constexpr int R = kRec<DIM, CONT>;
        const double2* const rec = reinterpret_cast<const double2*>(G.pf + (size_t)k * R);
#pragma unroll 4
        for (uint32_t s = 0; s < slots; s++) {
            const double2* const p = rec + s * n * (R / 2);
            const double2 f = p[0];
            ax += f.x;
            ay += f.y;
            if (R == 4) {
                const double2 g = p[R / 2 - 1];
                if (DIM == 3) az += g.x;
                if (CONT) rate += g.y;
            }
        }
        cnt = slots;
        if (more && G.itype[k] != P.type_non_existent) {
            D3 r, v;
            double rho, pr2;
            force_rows<DIM>(G, k, r, v, rho, pr2);
            const int32_t tk = G.itype[k];
            unstored_neighbours<DIM>(P, G, k, over, slots, [&](uint32_t i, D3 d, double d2) {
                D3 ri, vi;
                double rhoi, pri, ck, ci;
                force_rows<DIM>(G, i, ri, vi, rhoi, pri);
                const Kern kk = cubic_any(C, d2);
                force_coefs<DIM>(P, C, kk.s, d2, d, v, vi, rho, rhoi, pr2, pri, tk, G.itype[i], ck, ci);
                ax = fma(d.x, ck, ax);
                ay = fma(d.y, ck, ay);
                if (DIM == 3) az = fma(d.z, ck, az);
                if (CONT) {
                    double t, ti;
                    rate_terms<DIM>(P, C, G, k, i, kk.s, d2, d, t, ti);
                    rate += t;
                }
                cnt++;
            });
        }
        const uint32_t id = G.id[k];
        S.ax[id] = ax;
        S.ay[id] = ay;
        if (DIM == 3) S.az[id] = az;
        if (CONT) {
            S.drho[id] = rate;
            if (cnt > P.max_nb - 1) atomicOr(flags, RRSPH_FLAG_NEIGHBOUR_OVERFLOW);
        }
    }
    if (CONT) warp_sum_add(&scal->pairs, cnt);
}

}  // namespace

template <int DIM>
void launch_pair_masks(const DevParams& P, const State& S, const Sorted& G, StepScalars* scal, cudaStream_t st) {
    const unsigned extra = has_pistons(P, S) ? 1 : 0;
    k_pair_masks<DIM><<<(P.n + 31) / 32 + extra, 32 * Pm<DIM>::nc, 0, st>>>(P, S, G, scal);
}
template <int DIM>
void launch_pair_terms(const DevParams& P, const Sorted& G, cudaStream_t st, int threads) {
    const dim3 grid((P.n + threads - 1) / threads, pair_slices(P.n));
    const size_t sh = (size_t)(threads / 32) * 2 * kStack * sizeof(uint2);
    if (P.density_treatment != 0) k_pair_terms<DIM, true><<<grid, threads, sh, st>>>(P, G);
    else k_pair_terms<DIM, false><<<grid, threads, sh, st>>>(P, G);
}
template <int DIM>
void launch_pair_density(const DevParams& P, const State& S, const Sorted& G, StepScalars* scal, uint32_t* flags,
                         cudaStream_t st) {
    k_pair_density<DIM><<<(P.n + 127) / 128, 128, 0, st>>>(P, S, G, scal, flags);
}
template <int DIM>
void launch_pair_forces(const DevParams& P, const Sorted& G, cudaStream_t st, int threads) {
    const dim3 grid((P.n + threads - 1) / threads, pair_slices(P.n));
    const size_t sh = (size_t)(threads / 32) * (sizeof(Approach<DIM>) + kStack * sizeof(uint2));
    k_pair_forces<DIM><<<grid, threads, sh, st>>>(P, G);
}
template <int DIM>
void launch_pair_sum(const DevParams& P, const State& S, const Sorted& G, StepScalars* scal, uint32_t* flags,
                     cudaStream_t st) {
    if (P.density_treatment != 0) k_pair_sum<DIM, true><<<(P.n + 127) / 128, 128, 0, st>>>(P, S, G, scal, flags);
    else k_pair_sum<DIM, false><<<(P.n + 127) / 128, 128, 0, st>>>(P, S, G, scal, flags);
}

#define RRSPH_INSTANTIATE(D)                                                                                    \
    template void launch_pair_masks<D>(const DevParams&, const State&, const Sorted&, StepScalars*, cudaStream_t); \
    template void launch_pair_terms<D>(const DevParams&, const Sorted&, cudaStream_t, int);                     \
    template void launch_pair_density<D>(const DevParams&, const State&, const Sorted&, StepScalars*, uint32_t*, \
                                         cudaStream_t);                                                         \
    template void launch_pair_forces<D>(const DevParams&, const Sorted&, cudaStream_t, int);                    \
    template void launch_pair_sum<D>(const DevParams&, const State&, const Sorted&, StepScalars*, uint32_t*,    \
                                     cudaStream_t);
RRSPH_INSTANTIATE(2)
RRSPH_INSTANTIATE(3)
#undef RRSPH_INSTANTIATE

}  // namespace rrsph
