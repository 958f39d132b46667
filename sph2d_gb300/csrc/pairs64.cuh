// pairs64.cuh — the device code of the stored-pair FP64 sums that the step
// (kernels_pairs64.cu) and its adjoint (adjoint.cu) share: neighbour masks, roots
// and quotients, the walk that hands a warp 32 pairs at a time, and what is not stored.
#pragma once

#include <type_traits>

#include "kernels.cuh"
#include "neighbour.cuh"

namespace rrsph {

namespace {

template <int DIM>
struct Pm {  // masks of this dimension
    using T = typename std::conditional<DIM == 3, unsigned long long, uint32_t>::type;
    static constexpr uint32_t bits = DIM == 3 ? 64 : 32;
    static constexpr int nc = DIM == 3 ? 27 : 9;
    static __device__ __forceinline__ uint32_t popc(T m) {
        return DIM == 3 ? (uint32_t)__popcll((unsigned long long)m) : (uint32_t)__popc((uint32_t)m);
    }
    static __device__ __forceinline__ uint32_t lowest(T m) {
        return DIM == 3 ? (uint32_t)(__ffsll((long long)m) - 1) : (uint32_t)(__ffs((int)m) - 1);
    }
    static __device__ __forceinline__ T* masks(const Sorted& G) { return reinterpret_cast<T*>(G.nbmask); }
    static __device__ __forceinline__ T* nears(const Sorted& G) { return reinterpret_cast<T*>(G.pnear); }
};

// Cell c of the stencil of the cell `key` (in the order of
// get_neighbouring_cells2/3, GridUtils.h:190-250), stepping the interleaved
// coordinates in place; false where the reference drops the cell (a coordinate
// below 0 or above 65535, GridUtils.h:158-163, a key beyond the grid). wraps: a
// 3D coordinate of 1024 became 0 (GridUtils.h:50-64).
template <int DIM>
__device__ __forceinline__ bool stencil_cell(const DevParams& P, uint32_t key, int c, uint32_t& cell, bool& wraps) {
    constexpr uint32_t axis = DIM == 3 ? 0x09249249u : 0x55555555u;
    uint32_t out = 0;
    bool valid = true;
    wraps = false;
#pragma unroll
    for (int a = 0; a < DIM; a++) {
        const int d = DIM == 3 ? (a == 0 ? c / 9 : (a == 1 ? (c / 3) % 3 : c % 3)) - 1 : (a == 0 ? c / 3 : c % 3) - 1;
        const uint32_t m = axis << a, x = key & m;
        if (d < 0) valid = valid && x != 0;
        if (d > 0) {
            if (DIM == 3) wraps = wraps || x == m;
            else valid = valid && x != m;
        }
        const uint32_t up = ((x | ~m) + (1u << a)) & m, down = (x - (1u << a)) & m;
        out |= d < 0 ? down : (d > 0 ? up : x);
    }
    cell = out;
    return valid && out < P.max_cells;
}
// Displacement of stencil cell c, in cells.
template <int DIM>
__device__ __forceinline__ float3 stencil_shift(int c) {
    return DIM == 3 ? make_float3((float)(c / 9 - 1), (float)((c / 3) % 3 - 1), (float)(c % 3 - 1))
                    : make_float3((float)(c / 3 - 1), (float)(c % 3 - 1), 0.0f);
}

struct D3 {
    double x, y, z;
};
// Row k of a packed array of DIM (3D: padded to 4) doubles; .w the fourth.
template <int DIM>
__device__ __forceinline__ D3 row(const double* __restrict__ a, uint32_t k) {
    const double2 q = *reinterpret_cast<const double2*>(a + (size_t)k * (DIM == 3 ? 4 : 2));
    return {q.x, q.y, DIM == 3 ? a[(size_t)k * 4 + 2] : 0.0};
}
template <int DIM>
__device__ __forceinline__ D3 row4(const double* __restrict__ a, uint32_t k, double& w) {
    const double2* const p = reinterpret_cast<const double2*>(a + (size_t)k * 4);
    const double2 q = p[0], u = p[1];
    w = u.y;
    return {q.x, q.y, u.x};
}
// Position, and velocity with (rho, p / rho^2) of sorted particle k: in 2D three
// double2 rows, in 3D rho and p / rho^2 ride in the fourth words.
template <int DIM>
__device__ __forceinline__ void force_rows(const Sorted& G, uint32_t k, D3& r, D3& v, double& rho, double& pr2) {
    if (DIM == 3) {
        r = row4<3>(G.pr, k, rho);
        v = row4<3>(G.pv, k, pr2);
    } else {
        r = row<2>(G.pr, k);
        v = row<2>(G.pv, k);
        const double2 q = reinterpret_cast<const double2*>(G.pq)[k];
        rho = q.x;
        pr2 = q.y;
    }
}

// A double x > 0 scaled by a power of two to a float pair hi + lo (48 bits): hi
// gets the biased exponent ex, which the caller picks.
__device__ __forceinline__ void float_pair(double x, int ex, float& hi, float& lo) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    hi = __uint_as_float(((uint32_t)ex << 23) | ((uint32_t)(b >> 29) & 0x7FFFFFu));
    lo = (float)((uint32_t)b & 0x1FFFFFFFu) * __uint_as_float((uint32_t)(ex - 52) << 23);
}
// y0 (1 + c), y0 an approximation whose low word is zero, |c| < 2^-19: the
// mantissa is stepped as an integer in units of 2^-40 (at most 2^22 of them, what
// the rounding constant takes).
__device__ __forceinline__ double step_mantissa(double y0, float z, float c) {
    const float d = fmaf(z * c, 1099511627776.0f, 12582912.0f);  // z in [1, 2) is y0's mantissa; 2^40, 1.5 * 2^23
    const long long step = (long long)(__float_as_int(d) - 0x4B400000) << 12;
    return __longlong_as_double(__double_as_longlong(y0) + step);
}

// 1/sqrt(x) and 1/x to 2^-40 without the FP64 pipe: the approximation instruction
// (2^-20) and one third-order step in float pairs. The rest of the error is taken
// out by the caller with a second-order Newton step on what it wants,
//   d = x y:           sqrt(x) = d + (y/2)(x - d d)   (the residual is exact: half a unit)
//   eh = 1/2 - d (y/2): 1/sqrt(x) = y + y eh
//   e = 1 - x r:       v/x = v r + v r e
// so that a root takes three FP64 operations, its inverse two more, and a
// quotient three, where the IEEE forms take about eight each. The root of zero
// or a subnormal x (coincident particles) gives infinity.
__device__ __forceinline__ double inv_root_40(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const int hx = __double2hiint(x), hy = __double2hiint(y);
    const float z = __uint_as_float(0x3F800000u | ((uint32_t)hy & 0xFFFFFu) << 3);
    float mh, ml;  // x 2^(2k) with y = z 2^k: x y^2 = m z^2
    float_pair(x, (hx >> 20) + 2 * (hy >> 20) - 3 * 1023 + 127, mh, ml);  // x > 0
    const float p = z * z, pl = fmaf(z, z, -p);
    float e = fmaf(-mh, p, 1.0f);
    e = fmaf(-mh, pl, e);
    e = fmaf(-ml, p, e);
    const double r = step_mantissa(y, z, e * fmaf(0.375f, e, 0.5f));
    return hx < 0x00100000 ? y : r;
}
__device__ __forceinline__ double inverse_40(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const int hx = __double2hiint(x), hy = __double2hiint(y);
    const float z = __uint_as_float(0x3F800000u | ((uint32_t)hy & 0xFFFFFu) << 3);
    float mh, ml;
    float_pair(x, ((hx >> 20) & 0x7FF) + ((hy >> 20) & 0x7FF) - 2 * 1023 + 127, mh, ml);  // the sign is y's
    float e = fmaf(-mh, z, 1.0f);
    e = fmaf(-ml, z, e);
    return step_mantissa(y, z, fmaf(e, e, e));
}
// Infinite or not a number.
__device__ __forceinline__ bool no_number(double x) { return (__double2hiint(x) & 0x7FF00000) == 0x7FF00000; }
// Below zero; a NaN of either sign is not (the machine's own has the sign bit set).
__device__ __forceinline__ bool negative(double x) {
    return (uint32_t)__double2hiint(x) - 0x80000000u <= 0x7FF00000u;
}
// Half of a normal double, by its exponent.
__device__ __forceinline__ double half_of(double x) {
    return __hiloint2double(__double2hiint(x) - 0x00100000, __double2loint(x));
}

// The cubic spline at squared distance d2 (SmoothingKernel.h:20-56): m W, and
// m s with dW/dr = (r_i - r_j) s. NEAR: the branch q <= 1, which the masks' float
// test gives to all up to there and to some just beyond. These go through
// cubic_beyond (the branches' gradients differ by 2 (q - 1)^2, 1e-13 at the float
// test's error): a call, since the FP64 pipe would issue a few predicated operations
// for every pair.
struct Kern {
    double w, s;
};
__device__ __noinline__ Kern cubic_beyond(double w6, double s2, double q, double y1, double r) {
    const double y = fma(y1, fma(-r, half_of(y1), 0.5), y1);
    const double t = 2.0 - q, t2 = t * t;
    return {(w6 * t) * t2, (s2 * y) * t2};
}
// q >= 1
__device__ __forceinline__ bool beyond(double q) { return __double2hiint(q) >= 0x3FF00000; }
template <bool NEAR, bool W>
__device__ __forceinline__ Kern cubic(const PairConst& C, double d2) {
    const double y1 = inv_root_40(d2);
    const double r = d2 * y1;
    const double dist = fma(fma(-r, r, d2), half_of(y1), r);
    const double q = __double2hiint(y1) == 0x7FF00000 ? 0.0 : dist * C.inv_h;
    Kern k{0.0, 0.0};
    if (NEAR) {
        if (beyond(q)) return cubic_beyond(C.w6, C.s2, q, y1, r);
        if (W) k.w = fma(q * q, fma(C.w3, q, C.w2), C.w0q);
        k.s = fma(C.s1q, q, C.s1);
    } else {
        const double y = fma(y1, fma(-r, half_of(y1), 0.5), y1);
        const double t = 2.0 - q, t2 = t * t;
        const bool in = __double2hiint(t) >= 0;  // q <= 2
        if (W) k.w = in ? (C.w6 * t) * t2 : 0.0;
        k.s = in ? (C.s2 * y) * t2 : 0.0;
    }
    return k;
}

__device__ __forceinline__ double dot2(D3 a, D3 b) { return fma(a.x, b.x, a.y * b.y); }
template <int DIM>
__device__ __forceinline__ double dot(D3 a, D3 b) {
    return DIM == 3 ? fma(a.z, b.z, dot2(a, b)) : dot2(a, b);
}

// Pairs with a Lennard-Jones part: a fluid and a boundary particle.
__device__ __forceinline__ bool lj_pair(const DevParams& P, int32_t tk, int32_t ti) {
    return P.repulsive && ((tk > 0 && ti < 0) || (ti > 0 && tk < 0));
}

__device__ __forceinline__ double flip(double x) {
    return __hiloint2double(__double2hiint(x) ^ 0x80000000, __double2loint(x));
}
// The walk of the two pair passes: a warp takes 32 consecutive particles (and,
// of `slices` warps sharing them, every slices-th stencil cell), each lane hands
// out its particle's owned pairs (the neighbours with a larger sorted index) one
// at a time onto a small stack, and whenever 32 are there the warp evaluates
// them, one a lane. SPLIT: two stacks, for the two branches of the kernel, so
// that a warp runs one of them. ORD: number the owned pairs of a particle too.
// All lanes call f(word pair, lane has a pair, near as a constant) together;
// pair_of() reads the words.
constexpr int kStack = 64;  // up to 31 waiting and 32 pushed
struct Pair {
    uint32_t k, i;   // sorted indices, k < i
    uint32_t rank;   // i's number among k's neighbours (255: that or more)
    uint32_t order;  // and among the owned ones
    int c;           // i's cell in k's stencil
    uint32_t bit;    // k's bit in its own cell
};
// k0: the first particle of the warp.
__device__ __forceinline__ Pair pair_of(uint2 e, uint32_t k0) {
    return {k0 + (e.y & 31u), e.x, (e.y >> 16) & 255u, e.y >> 24, (int)((e.y >> 5) & 31u), (e.y >> 10) & 63u};
}
__device__ __forceinline__ uint32_t warp_first() { return (blockIdx.x * blockDim.x + threadIdx.x) & ~31u; }
template <int DIM, bool SPLIT, bool ORD, class F>
__device__ __forceinline__ void walk_pairs(const DevParams& P, const Sorted& G, uint2* stacks, F&& f) {
    using M = Pm<DIM>;
    using T = typename M::T;
    const uint32_t lane = threadIdx.x & 31u, below = (1u << lane) - 1u;
    const uint32_t k0 = warp_first(), k = k0 + lane;
    if (k0 >= P.n) return;
    uint2* const far_stack = stacks + (threadIdx.x >> 5) * (SPLIT ? 2 * kStack : kStack);
    uint2* const near_stack = far_stack + kStack;
    const int step = (int)gridDim.y;
    const size_t n = P.n;
    // a particle whose own cell is searched in place stores nothing
    const bool active = k < P.n && !((M::masks(G)[(size_t)M::nc * n + k] >> (M::nc / 2)) & 1u);
    const uint32_t bit = active ? k - G.pfirst[(size_t)(M::nc / 2) * n + k] : 0u;
    // the lanes go through the cells together, the next cell's words loaded ahead
    // (each lane at its own pace, a load after another by some lane in most rounds,
    // took 165 us for the 2D terms of the 409k flume and 2.4 ms for 385k in 3D)
    T m_next = 0, close_next = 0;
    uint32_t first_next = 0, before_next = 0, own_next = 0;
    auto fetch = [&](int c) {
        m_next = 0;
        if (!active || c >= M::nc) return;
        const size_t at = (size_t)c * n + k;
        m_next = M::masks(G)[at];
        first_next = G.pfirst[at];
        before_next = G.pbefore[at];
        if (SPLIT) close_next = M::nears(G)[at];
        if (ORD) own_next = G.pown[at];
    };
    uint32_t held = 0, held_near = 0;
    fetch((int)blockIdx.y);
    for (int c = (int)blockIdx.y; c < M::nc; c += step) {
        const T all = m_next, close = close_next;
        const uint32_t first = first_next, before = before_next;
        uint32_t order = own_next;
        fetch(c + step);
        T bits = all;
        if (c == M::nc / 2) bits &= ~(((T)2 << bit) - 1);  // without itself and the particles before it
        else if (first < k) bits = 0;
        for (;;) {
            const bool has = bits != 0;
            bool near = false;
            uint2 e;
            if (has) {
                const uint32_t b = M::lowest(bits);
                const T lower = ((T)1 << b) - 1;
                bits &= bits - 1;
                near = SPLIT && ((close >> b) & 1u);
                const uint32_t rank = min(before + M::popc(all & lower), 255u);
                e = make_uint2(first + b, lane | (uint32_t)c << 5 | bit << 10 | rank << 16 | min(order, 255u) << 24);
                order++;
            }
            const uint32_t who = __ballot_sync(0xFFFFFFFFu, has && !near);
            const uint32_t who_near = SPLIT ? __ballot_sync(0xFFFFFFFFu, near) : 0u;
            if ((who | who_near) == 0) break;
            if (has) {
                if (near) near_stack[held_near + __popc(who_near & below)] = e;
                else far_stack[held + __popc(who & below)] = e;
            }
            held += __popc(who);
            held_near += __popc(who_near);
            __syncwarp();
            if (held >= 32) {
                held -= 32;
                f(far_stack[held + lane], true, std::false_type{});
                __syncwarp();
            }
            if (SPLIT && held_near >= 32) {
                held_near -= 32;
                f(near_stack[held_near + lane], true, std::true_type{});
                __syncwarp();
            }
        }
    }
    f(far_stack[lane], lane < held, std::false_type{});
    if (SPLIT) f(near_stack[lane], lane < held_near, std::true_type{});
}

// The rank of k among i's neighbours: k is bit `bit` of i's stencil cell opposite c.
template <int DIM>
__device__ __forceinline__ uint32_t rank_of(const DevParams& P, const Sorted& G, uint32_t i, int c, uint32_t bit) {
    using M = Pm<DIM>;
    const size_t at = (size_t)(M::nc - 1 - c) * P.n + i;
    const typename M::T m = M::masks(G)[at];
    return G.pbefore[at] + M::popc(m & (((typename M::T)1 << bit) - 1));
}

// The kernel of a pair that stores none.
__device__ __forceinline__ Kern cubic_any(const PairConst& C, double d2) {
    return d2 < C.h * C.h ? cubic<true, true>(C, d2) : cubic<false, true>(C, d2);
}

// The neighbours of k whose values are not stored: ranks from `first` on, and
// the cells searched in place. f(i, r_i - r_k, squared distance).
template <int DIM, class F>
__device__ __forceinline__ void unstored_neighbours(const DevParams& P, const Sorted& G, uint32_t k, uint32_t over,
                                                    uint32_t first, F&& f) {
    using M = Pm<DIM>;
    const uint32_t key = G.key[k];
    const D3 a = row<DIM>(G.pr, k);
    uint32_t rank = 0;
    for (int c = 0; c < M::nc; c++) {
        uint32_t cell;
        bool wraps;
        if ((over >> c) & 1u) {
            stencil_cell<DIM>(P, key, c, cell, wraps);
            for (uint32_t i = G.cell_start[cell]; i < G.cell_end[cell]; i++) {
                if (i == k || G.itype[i] == P.type_non_existent) continue;
                const D3 b = row<DIM>(G.pr, i);
                const D3 d{__dsub_rn(b.x, a.x), __dsub_rn(b.y, a.y), DIM == 3 ? __dsub_rn(b.z, a.z) : 0.0};
                const double d2 = exact_dist2<DIM>(d.x, d.y, d.z);
                if (d2 < P.cut2) f(i, d, d2);
            }
            continue;
        }
        typename M::T m = M::masks(G)[(size_t)c * P.n + k];
        if (m == 0) continue;
        const uint32_t base = G.pfirst[(size_t)c * P.n + k];
        for (; m; m &= m - 1, rank++) {
            if (rank < first) continue;
            const uint32_t i = base + M::lowest(m);
            const D3 b = row<DIM>(G.pr, i);
            const D3 d{b.x - a.x, b.y - a.y, DIM == 3 ? b.z - a.z : 0.0};
            f(i, d, dot<DIM>(d, d));
        }
    }
}

// What of k's neighbours is stored: the number of slots; whether others remain.
template <int DIM>
__device__ __forceinline__ bool stored_slots(const DevParams& P, const Sorted& G, uint32_t k, uint32_t& over,
                                             uint32_t& slots) {
    using M = Pm<DIM>;
    over = (uint32_t)M::masks(G)[(size_t)M::nc * P.n + k];
    const uint32_t cnt = G.pcount[k];
    slots = (over >> (M::nc / 2)) & 1u ? 0u : min(cnt, P.pc.cap);
    return over != 0 || cnt > slots;
}

// Warps that share 32 particles' stencil cells in the pair passes: one where the
// particles alone give every SM a dozen warps; a third or a ninth of the cells
// each below that, where one warp's pairs in a row would be the whole step's time.
int pair_slices(uint32_t n) {
    const uint32_t warps = (n + 31) / 32;
    return warps >= 1824 ? 1 : (warps >= 608 ? 3 : 9);
}

}  // namespace

}  // namespace rrsph
