// kernels_reuse.cu — the FP32-mixed step with neighbour reuse: candidate
// lists kept between grid builds, the density gather over them (which writes
// the step's neighbour list) and the force gather over that list with the
// whole step fused in. 2D and 3D, summation and continuity density.
//
// A particle's candidate list holds the particles within cutoff + skin of it
// when the grid was last built; while no particle has moved more than skin/2
// since then, every pair within the cutoff is in the lists, and each step
// tests the list instead of the 3^dim stencil cells (the pair set is the
// reference's: the same cutoff test).
//
// Positions are fixed point, kFixOne units a cell, modulo 2^32 (kernels.cuh,
// Pos): the separation of two particles within 16 cells of each other is the
// difference of their words whatever cells they are in, so a list entry is a bare
// index and a pair's separation costs a subtraction and a conversion per axis.
// The density pass writes the candidates that are neighbours as a second list for
// the force pass, four entries a store. (Cell-relative floats with a cell code per
// entry, decoded by both passes, and single-word list stores took 95 and 100
// instructions a pair, and the stores three quarters of the density pass's L2
// traffic. One bit a candidate instead of a second list left the force gather
// with 23 of 32 lanes: 68 us on the flume.) us per step, before and after: 409k
// flume 123.6 / 116, 1.06M 3D dam break 824 / 718, 928k ensemble 254 / 235, 43k
// delta-SPH dam break 39.4 / 36.1. The 16-byte neighbour loads bound both passes
// now: L1 79 % busy in the density pass, loads in flight in the force pass.
#include "reuse.cuh"

namespace rrsph {

namespace {

constexpr int kVlBatch = 4;       // list entries the density gather loads together (one uint4)
// neighbours the force gather loads together: four for the 2D common method
// set, two elsewhere (four would spill the registers of the general pair)
template <int DIM, bool STD>
constexpr int kVlForceBatch = DIM == 2 && STD ? 4 : 2;

template <int DIM>
struct Vl {
    static constexpr int cap = DIM == 3 ? kVerletCap3 : kVerletCap2;
    static constexpr uint32_t cmax = DIM == 3 ? 0x3FFu : kMaxCellCoord2;  // largest cell coordinate of a key
};

// The split gathers (L > 1): a block of L warps takes 32 particles, warp `sub`
// their list groups sub, sub + L, ..., and the first warp adds the partial sums up
// and goes on alone. With few particles a thread walking its whole list is one
// long chain of dependent loads on a nearly empty chip.
// A warp's neighbours go to the slab groups it reads (sub + L j), so no warp waits
// for another's count; the L counts share the particle's word.
template <int L>
constexpr uint32_t kCountBits = 32 / L;
template <int L>
__device__ __forceinline__ uint32_t sub_count(uint32_t word, uint32_t sub) {
    return L == 1 ? word : (word >> (sub * kCountBits<L>)) & ((1u << (kCountBits<L> & 31u)) - 1u);
}
// The word of a list of c entries stored in consecutive groups.
template <int L>
__device__ __forceinline__ uint32_t packed_counts(uint32_t c) {
    if (L == 1) return c;
    uint32_t word = 0;
    for (uint32_t g = 0; 4 * g < c; g++) word += min(4u, c - 4 * g) << ((g % L) * kCountBits<L>);
    return word;
}

// Separation of two positions in fixed-point units, exact before the conversion ...
template <int DIM>
__device__ __forceinline__ float3 difference(const Pos& i, const Pos& j) {
    auto diff = [](int a, int b) { return (float)(int)((uint32_t)a - (uint32_t)b); };
    return make_float3(diff(i.x, j.x), diff(i.y, j.y), DIM == 3 ? diff(i.z, j.z) : 0.0f);
}
// ... and in metres.
template <int DIM>
__device__ __forceinline__ float3 separation(const Pos& i, const Pos& j, float u) {
    const float3 d = difference<DIM>(i, j);
    return make_float3(d.x * u, d.y * u, DIM == 3 ? d.z * u : 0.0f);
}
// Squared distance, + the neighbour's code: nothing for a live particle, infinite
// or NaN (never below a cutoff) for one that is absent or not listed.
template <int DIM>
__device__ __forceinline__ float distance2(float3 d, float code) {
    return DIM == 3 ? fmaf(d.x, d.x, fmaf(d.y, d.y, fmaf(d.z, d.z, code))) : fmaf(d.x, d.x, fmaf(d.y, d.y, code));
}
// The reference's cutoff test in double (inside the guard band, and for a
// particle outside the grid): rare, so the positions come from the id-order state.
template <int DIM>
__device__ __noinline__ bool exact_pair(const DevParams& P, const State& S, uint32_t a, uint32_t b) {
    const double dx = __dsub_rn(S.rx[a], S.rx[b]), dy = __dsub_rn(S.ry[a], S.ry[b]);
    const double dz = DIM == 3 ? __dsub_rn(S.rz[a], S.rz[b]) : 0.0;
    return exact_dist2<DIM>(dx, dy, dz) < P.cut2;
}
// The stencil search's test of particle i (sorted) against k: an absent one never,
// in double one outside the grid and those of a cell that the stencil meets by
// wrapping (the 3D key of coordinate 1024 is that of 0, 1024 cells away, where fixed
// point repeats).
template <int DIM>
__device__ __forceinline__ bool searched_pair(const DevParams& P, const State& S, const Sorted& G, uint32_t i,
                                              uint32_t k, const Pos& pi, const Pos& pk, bool wraps) {
    if (pi.absent()) return false;
    if (wraps || pi.unlisted() || pk.unlisted()) return exact_pair<DIM>(P, S, G.id[i], G.id[k]);
    const float d2 = distance2<DIM>(separation<DIM>(pi, pk, P.rf.u), pi.code);
    if (d2 < P.mf.cut2_lo) return true;
    return d2 < P.mf.cut2_hi && exact_pair<DIM>(P, S, G.id[i], G.id[k]);
}

// Whether a stencil cell with these offsets is met by wrapping.
template <int DIM>
__device__ __forceinline__ bool wrapped(int sx, int sy, int sz) {
    return DIM == 3 && (sx < -1 || sy < -1 || sz < -1);
}

__device__ __forceinline__ float rcp_approx(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
// The cubic spline, zero beyond q = 2 (cells may be wider): W / f with q = |r| / h ...
__device__ __forceinline__ float cubic_w(float q) {
    const float t = fmaxf(2.0f - q, 0.0f);
    const float far = (1.0f / 6.0f) * (t * (t * t));
    const float near = fmaf(q * q, fmaf(0.5f, q, -1.0f), 2.0f / 3.0f);
    return q <= 1.0f ? near : far;
}
// ... and s with dW/dr = diff s f / (2 h^2) (rs: 1 / distance).
__device__ __forceinline__ float cubic_s(const ReuseF& U, float q, float rs) {
    const float t = fmaxf(2.0f - q, 0.0f);
    const float far = -(rs * U.far) * (t * t);
    const float near = fmaf(3.0f, q, -4.0f);
    return q <= 1.0f ? near : far;
}
// A compensated sum times a factor, as an unevaluated sum of two floats.
__device__ __forceinline__ F2 scaled(const Kahan& a, F2 f) {
    const float hi = a.s * f.hi;
    return {hi, fmaf(a.s, f.hi, -hi) + (a.s * f.lo - a.c * f.hi)};
}
__device__ __forceinline__ double value(F2 v) { return f2d(v.hi) + f2d(v.lo); }

__global__ void k_vl_decide(cudaGraphConditionalHandle h, const uint32_t* __restrict__ rebuild) {
    cudaGraphSetConditional(h, *rebuild ? 1u : 0u);
}
__global__ void k_vl_reset(uint32_t* __restrict__ rebuild, uint32_t* __restrict__ gone,
                           uint32_t* __restrict__ far, unsigned long long* __restrict__ builds) {
    *rebuild = 0u;
    *gone = 0u;
    far[1] = far[0];  // for this rebuild; the next key pass raises its own
    far[0] = 0u;
    *builds += 1ull;
}
// After an upload: a flag raised by the key pass that ran for the replaced
// positions is dropped (the next key pass checks the uploaded ones), unless no
// list exists yet (all bits set) or the last build left out a non-existent
// particle or overflowed a list.
__global__ void k_vl_upload_check(uint32_t* __restrict__ rebuild, const uint32_t* __restrict__ gone) {
    if (*rebuild != 0xFFFFFFFFu) *rebuild = *gone ? 1u : 0u;
}

// The window of cell offsets along one axis a particle at offset p from its
// cell's lower edge searches: the cell equals the cutoff and the skin is at
// most h, so a candidate within cutoff + skin lies at most two cells away, and
// two only on the side whose edge is within one skin.
template <int DIM>
__device__ __forceinline__ void vl_window(float p, uint32_t c, float cell, float edge, int& lo, int& hi) {
    lo = (p < edge && c >= 2) ? -2 : (c >= 1 ? -1 : 0);
    hi = (p > cell - edge && c + 2 <= Vl<DIM>::cmax) ? 2 : (c + 1 <= Vl<DIM>::cmax ? 1 : 0);
}

// Distance along one axis from a particle at offset p in [0, cell] from its
// cell's lower edge to the nearest side of the cell d cells away.
__device__ __forceinline__ float gap_to_cell(int d, float p, float cell) {
    return d > 0 ? (float)d * cell - p : (d < 0 ? p - (float)(d + 1) * cell : 0.0f);
}

// After this step's grid (sort + reorder): each particle's candidates, four
// entries gathered in registers and stored as one uint4 into the group's slab
// (the lanes of a warp store neighbouring uint4s), in cell order x outer, the last
// group padded with the row of an absent particle (index n). A particle outside
// the grid gets no list: it is searched, as is one with too many candidates.
//
// A thread first lists the cells of its window, then goes through their particles
// in one loop: a warp's lanes then wait for the lane with the most particles, not
// in every cell for the lane whose cell holds most (half of the lanes were idle).
// The entries pass through a ring in shared memory, as in the density pass: no
// branch per candidate. us a rebuild, walking cell by cell and so: 409k flume 96 / 88,
// 43k dam break 31 / 22, 1.06M in 3D 1014 / 725.
constexpr int kVlBuildThreads = 128;
constexpr int kVlRow = 5;  // cells along an axis of the window, at most
template <int DIM>
__global__ void __launch_bounds__(kVlBuildThreads) k_vl_build(DevParams P, State S, Sorted G) {
    constexpr int CAP = Vl<DIM>::cap;
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= P.n) return;
    const ReuseF& U = P.rf;
    const float cell = P.mf.cell;
    const uint32_t id = G.id[k], key = G.key[k];
    const Pos pj = G.pos[k];
    uint32_t cx, cy, cz = 0;
    if (DIM == 3) {
        cx = third_bits(key);
        cy = third_bits(key >> 1);
        cz = third_bits(key >> 2);
        S.bfix4[id] = make_int4(pj.x, pj.y, pj.z, (int)(cx | cy << 10 | cz << 20));
    } else {
        cx = second_bits(key);
        cy = second_bits(key >> 1);
        S.bfix2[id] = make_int2(pj.x, pj.y);
        S.bcxy[id] = cx | cy << 16;
    }
    S.slot[id] = k;
    uint4* const slab = reinterpret_cast<uint4*>(G.vlist) + k;  // group g at slab[g * n]
    // this thread's columns: the non-empty cells of a row of its window, as ranges of
    // sorted indices, and a ring of eight list entries waiting to be stored
    __shared__ uint2 ranges[kVlRow][kVlBuildThreads];
    __shared__ uint32_t ring[8][kVlBuildThreads];
    const uint32_t t = threadIdx.x;
    uint32_t nl = 0, stored = 0;
    auto store4 = [&]() {
        const uint32_t q = stored & 4u;
        if (stored < (uint32_t)CAP)
            slab[(size_t)(stored >> 2) * P.n] = make_uint4(ring[q][t], ring[q + 1][t], ring[q + 2][t], ring[q + 3][t]);
        stored += 4;
    };
    if (pj.absent()) atomicOr(S.vl_gone, 1u);
    // offset from the lower edges of the key's cell
    const float px = (float)(int)((uint32_t)pj.x - (cx << kFixBits)) * U.u;
    const float py = (float)(int)((uint32_t)pj.y - (cy << kFixBits)) * U.u;
    const float pz = DIM == 3 ? (float)(int)((uint32_t)pj.z - (cz << kFixBits)) * U.u : 0.0f;
    // searched: a particle outside the grid, which no list holds, and where there is
    // one also those less than a cell below the grid's edge, which may meet it
    const bool outside = !pj.absent() && (pj.unlisted() || (S.vl_far[1] && (px < 0.0f || py < 0.0f || pz < 0.0f)));
    if (!pj.absent() && !outside) {
        const float edge = P.vl_skin_edge;
        int x0, x1, y0, y1, z0 = 0, z1 = 0;
        vl_window<DIM>(px, cx, cell, edge, x0, x1);
        vl_window<DIM>(py, cy, cell, edge, y0, y1);
        if (DIM == 3) vl_window<DIM>(pz, cz, cell, edge, z0, z1);
        const float cut = P.vl_cut2 / (U.u * U.u);
        uint32_t nr = 0;
        // notes the particles of cell c, if a point of it lies within the list cutoff
        // of the particle: the distances to its nearest sides, per axis, squared and
        // summed (the window's corner and far diagonal cells mostly hold no candidate)
        auto note = [&](uint32_t c, float gap2) {
            if (gap2 >= P.vl_cut2 || c >= P.max_cells) return;
            const uint32_t s = G.cell_start[c];
            if (s != kEmpty) ranges[nr++][t] = make_uint2(s, G.cell_end[c]);
        };
        // the noted particles four at a time, their loads together (the rows past a
        // cell's end are another cell's, or the spare ones past the last: skipped)
        auto candidates = [&]() {
            uint32_t r = 0, i0 = 0, e = 0;
            while (true) {
                if (i0 >= e) {
                    if (r == nr) break;
                    const uint2 se = ranges[r++][t];
                    i0 = se.x;
                    e = se.y;
                }
                const Pos* const row = G.pos + i0;
                Pos q[kVlBatch];
#pragma unroll
                for (int u = 0; u < kVlBatch; u++) q[u] = row[u];
#pragma unroll
                for (int u = 0; u < kVlBatch; u++) {
                    const uint32_t i = i0 + u;
                    const bool in = distance2<DIM>(difference<DIM>(q[u], pj), q[u].code) < cut && i < e && i != k;
                    if (in) ring[nl & 7u][t] = i;
                    nl += in;
                }
                if (nl - stored >= 4) store4();
                i0 += kVlBatch;
            }
            nr = 0;
        };
        auto square = [](float x) { return x * x; };
        if (DIM == 3) {
            const uint32_t mz0 = split3_32(cz + z0);
#pragma unroll 1
            for (int dx = x0; dx <= x1; dx++) {
                const uint32_t mx = split3_32(cx + dx);
                const float gx = square(gap_to_cell(dx, px, cell));
#pragma unroll 1
                for (int dy = y0; dy <= y1; dy++) {
                    const float gxy = gx + square(gap_to_cell(dy, py, cell));
                    if (gxy >= P.vl_cut2) continue;
                    const uint32_t mxy = mx | (split3_32(cy + dy) << 1);
                    uint32_t mz = mz0;
#pragma unroll 1
                    for (int dz = z0; dz <= z1; dz++) {
                        note(mxy | (mz << 2), gxy + square(gap_to_cell(dz, pz, cell)));
                        mz = ((mz | 0xF6DB6DB6u) + 1u) & 0x09249249u;  // of the next z
                    }
                    candidates();
                }
            }
        } else {
            const uint32_t my0 = split2_32(cy + y0);
#pragma unroll 1
            for (int dx = x0; dx <= x1; dx++) {
                const uint32_t mx = split2_32(cx + dx);
                const float gx = square(gap_to_cell(dx, px, cell));
                uint32_t my = my0;
#pragma unroll 1
                for (int dy = y0; dy <= y1; dy++) {
                    note(mx | (my << 1), gx + square(gap_to_cell(dy, py, cell)));
                    my = ((my | 0xAAAAAAAAu) + 1u) & 0x55555555u;  // of the next y
                }
                candidates();
            }
        }
    }
    if (nl > stored) {  // the last group, padded
        for (uint32_t u = nl; u < stored + 4; u++) ring[u & 7u][t] = P.n;
        store4();
    }
    const bool search = outside || nl > (uint32_t)CAP;
    G.vcount[k] = search ? kListOver : nl;
    if (search) {  // needs a fresh grid each step
        atomicOr(S.vl_rebuild, 1u);
        atomicOr(S.vl_gone, 2u);
    }
}

// One neighbour's term of the density gather, to be multiplied by term_factor():
// W (summation) or the continuity rate with its delta-SPH term (density_con,
// Density.h:63-114).
template <int DIM, int SKF, bool CONT>
__device__ __forceinline__ float density_term(const DevParams& P, float3 d, float d2, float4 vdi, float4 vdj) {
    const MixedF& M = P.mf;
    const ReuseF& U = P.rf;
    const float rs = inv_distance(d2);
    const float q = d2 * rs * M.inv_h;
    const int skf = SKF ? SKF : P.density_skf;
    if (!CONT) return SKF == 1 ? cubic_w(q) : kernel_wf(skf, M.kf[skf], q);
    const float sc = SKF == 1 ? cubic_s(U, q, rs) : kernel_dwdr_scalef(skf, M.kf[skf], q, rs, M.inv_h);
    float vcc = (vdi.x - vdj.x) * d.x + (vdi.y - vdj.y) * d.y;
    if (DIM == 3) vcc += (vdi.z - vdj.z) * d.z;
    float term = vcc * sc;
    if (P.density_treatment == 2) {
        const float rho_factor = __fdividef(vd4_drho<DIM>(vdi, vdj), M.rho0 + vdi.w);
        // (never false: with the select the 3D gather takes 64 registers, without 75 and 139k
        // particles 141 us a step instead of 133)
        term -= d2 >= 0.0f ? 2.0f * M.dhc * (rho_factor * sc) : 0.0f;
    }
    return term;
}
template <int SKF, bool CONT>
__device__ __forceinline__ F2 term_factor(const ReuseF& U) {
    return SKF != 1 ? U.m : (CONT ? U.a : U.w);
}

// density_sum (Density.h:25-61) + EOS, or density_con (Density.h:63-114), over
// the candidate list; the candidates within the cutoff are this step's
// neighbours, written to nlist for the force pass. A particle that is searched
// instead (the grid is rebuilt every step while one is) writes its neighbours too.
template <int DIM, int SKF, bool CONT, int L>
__global__ void __launch_bounds__(kMaxGatherThreads) k_density_verlet(DevParams P, State S, Sorted G,
                                                                     StepScalars* __restrict__ scal,
                                                                     uint32_t* __restrict__ flags) {
    constexpr int CAP = Vl<DIM>::cap;
    // the force gather may launch now: it waits for this grid at its start (griddepcontrol.wait)
    asm volatile("griddepcontrol.launch_dependents;");
    if (L > 1 && blockIdx.x * 32u >= P.n) {  // the extra block
        piston_block(P, S, scal);
        return;
    }
    const uint32_t lane = threadIdx.x & 31u, sub = L > 1 ? threadIdx.x >> 5 : 0u;
    const uint32_t k = L > 1 ? blockIdx.x * 32u + lane : blockIdx.x * blockDim.x + threadIdx.x;
    const bool active = k < P.n;
    uint32_t cnt = 0, word = 0;
    Kahan acc{0.0f, 0.0f};
    if (active) {
        const float u = P.rf.u, lo = P.mf.cut2_lo, hi = P.mf.cut2_hi;
        const Pos pj = G.pos[k];
        const float4 vdj = CONT ? G.VD4[k] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        const uint32_t vc = pj.absent() ? 0u : G.vcount[k];
        if (vc != kListOver) {
            const uint4* const slab = reinterpret_cast<const uint4*>(G.vlist) + k;  // group g at slab[g * n]
            const uint32_t groups = (vc + 3u) >> 2;
            // groups of four entries (one load, the next group's issued before this
            // one's particles are loaded), then their particles, loaded together; the
            // body has no branch but the rare guard-band test, and each group's sum is
            // added with compensation (list words are read once a step: streaming
            // loads keep L1 for the neighbours' data)
            // neighbours wait in a ring of eight words in shared memory until there are
            // four to store: no branch per candidate
            uint4* const out = reinterpret_cast<uint4*>(G.nlist) + (size_t)sub * P.n + k;  // this warp's group j at out[L j n]
            extern __shared__ uint32_t list_ring[];
            uint32_t* const ring = list_ring + threadIdx.x;  // word e & 7 at ring[(e & 7) blockDim.x]
            uint32_t stored = 0;
            auto store4 = [&]() {
                const uint32_t* const q = ring + (stored & 4u) * blockDim.x;
                out[(size_t)(L * (stored >> 2)) * P.n] = make_uint4(q[0], q[blockDim.x], q[2 * blockDim.x], q[3 * blockDim.x]);
                stored += 4;
            };
            uint4 w = make_uint4(P.n, P.n, P.n, P.n);
            if (sub < groups) w = __ldcs(slab + (size_t)sub * P.n);
            for (uint32_t g = sub; g < groups; g += L) {
                    const uint4 wn = g + L < groups ? __ldcs(slab + (size_t)(g + L) * P.n) : w;
                    const uint32_t en[kVlBatch] = {w.x, w.y, w.z, w.w};
                    Pos pb[kVlBatch];
#pragma unroll
                    for (int j = 0; j < kVlBatch; j++) pb[j] = G.pos[en[j]];
                    float3 d[kVlBatch];
                    float d2[kVlBatch];
                    bool in[kVlBatch], band = false;
#pragma unroll
                    for (int j = 0; j < kVlBatch; j++) {
                        d[j] = separation<DIM>(pb[j], pj, u);
                        d2[j] = distance2<DIM>(d[j], pb[j].code);
                        in[j] = d2[j] < lo;
                        band = band || (!in[j] && d2[j] < hi);
                    }
                    if (band) {
#pragma unroll 1
                        for (int j = 0; j < kVlBatch; j++) {
                            const float x = j == 0 ? d2[0] : (j == 1 ? d2[1] : (j == 2 ? d2[2] : d2[3]));
                            const uint32_t e = j == 0 ? en[0] : (j == 1 ? en[1] : (j == 2 ? en[2] : en[3]));
                            if (!(x < lo) && x < hi && exact_pair<DIM>(P, S, G.id[e], G.id[k])) {
                                if (j == 0) in[0] = true;
                                if (j == 1) in[1] = true;
                                if (j == 2) in[2] = true;
                                if (j == 3) in[3] = true;
                            }
                        }
                    }
                    float part = 0.0f;
#pragma unroll
                    for (int j = 0; j < kVlBatch; j++) {
                        const float4 vdi = CONT && in[j] ? G.VD4[en[j]] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                        const float t = density_term<DIM, SKF, CONT>(P, d[j], d2[j], vdi, vdj);
                        part += in[j] ? t : 0.0f;
                        if (in[j]) ring[(cnt & 7u) * blockDim.x] = en[j];
                        cnt += in[j];
                    }
                    if (cnt - stored >= 4) store4();
                    acc.add(part);
                    w = wn;
            }
            if (cnt > stored) store4();  // (the words past cnt are not read)
            word = cnt;
        } else if (sub == 0) {
            // the stencil search (the grid is this step's)
            uint32_t* const list = G.nlist + (size_t)k * 4;
            constexpr int NC = DIM == 3 ? 27 : 9;
            const Stencil<DIM> st(P, G.key[k]);
#pragma unroll 1
            for (int c = 0; c < NC; c++) {
                uint32_t cell;
                int sx, sy, sz;
                if (!st.cell(c, cell, sx, sy, sz)) continue;
                const uint32_t s = G.cell_start[cell];
                if (s == kEmpty) continue;
                const uint32_t e = G.cell_end[cell];
                const bool wraps = wrapped<DIM>(sx, sy, sz);
                float part = 0.0f;
                for (uint32_t i = s; i < e; i++) {
                    if (i == k) continue;
                    const Pos pi = G.pos[i];
                    if (!searched_pair<DIM>(P, S, G, i, k, pi, pj, wraps)) continue;
                    if (cnt < (uint32_t)CAP) list[(size_t)(cnt >> 2) * 4 * P.n + (cnt & 3u)] = i;
                    cnt++;
                    const float4 vdi = CONT ? G.VD4[i] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    const float3 d = separation<DIM>(pi, pj, u);
                    part += density_term<DIM, SKF, CONT>(P, d, distance2<DIM>(d, 0.0f), vdi, vdj);
                }
                acc.add(part);
            }
            word = packed_counts<L>(min(cnt, (uint32_t)CAP));
        }
    }
    if (L > 1) {
        __shared__ float ps[L][32], pc[L][32];
        __shared__ uint32_t pn[L][32];
        ps[sub][lane] = acc.s;
        pc[sub][lane] = acc.c;
        pn[sub][lane] = cnt;
        __syncthreads();
        if (sub != 0) return;
#pragma unroll
        for (int u = 1; u < L; u++) {  // (a searched particle's other warps counted nothing)
            acc.add(ps[u][lane]);
            acc.c += pc[u][lane];
            cnt += pn[u][lane];
            word += pn[u][lane] << ((uint32_t)u * kCountBits<L>);
        }
    }
    if (active) {
        const MixedF& M = P.mf;
        const uint32_t id = G.id[k];
        G.ncount[k] = word;
        if (cnt > P.max_nb - 1) atomicOr(flags, RRSPH_FLAG_NEIGHBOUR_OVERFLOW);
        if (!CONT) {
            // rho - rho0 = sum - (rho0 - m W(0)): the two are within a factor of two,
            // so the float difference is exact; the Kahan and rounding residuals follow
            const F2 sum = scaled(acc, term_factor<SKF, CONT>(P.rf));
            const float d = ((sum.hi - M.rho0_minus_w0_hi) + sum.lo) - M.rho0_minus_w0_lo;
            const float rho = M.rho0 + d;
            const float pr = eos_pf(M, d);
            const float2 prr = make_float2(pr, pr * __frcp_rn(rho * rho));
            if (DIM == 2)  // V4.zw = (the pressure the 2D force pass reads of a neighbour: p (form 1) or p/rho^2, rho)
                reinterpret_cast<float2*>(G.V4 + k)[1] = make_float2(P.intf_form == 1 ? prr.x : prr.y, rho);
            else
                G.V4[k].w = rho;
            G.PR[k] = prr;
            S.rho[id] = P.rho0 + f2d(d);
            S.p[id] = f2d(pr);
        } else {
            const float d = (float)(S.rho[id] - P.rho0);
            const float pr = eos_pf(M, d);
            const float rf = G.V4[k].w;  // rho_predict, the density of the forces
            const float2 prr = make_float2(pr, pr * __frcp_rn(rf * rf));
            if (DIM == 2) G.V4[k].z = P.intf_form == 1 ? prr.x : prr.y;
            G.PR[k] = prr;
            S.p[id] = pr;
            S.drho[id] = value(scaled(acc, term_factor<SKF, CONT>(P.rf)));
        }
    }
    warp_sum_add(&scal->pairs, cnt);
}

// One neighbour's coefficient of the separation in the acceleration, for the
// common method set (pressure form 2, Monaghan viscosity, cubic kernel, no
// artificial pressure or XSPH), over the factor ReuseF::a:
// s (p_i/rho_i^2 + p_j/rho_j^2 + Pi), one quotient for the two of the viscosity.
// lj: a boundary neighbour of a fluid particle under Lennard-Jones. MU: keep the
// largest |mu|.
template <int DIM, bool MU>
__device__ __forceinline__ float pair_coef(const DevParams& P, float3 d, float d2, const float4& vj, const float4& vi,
                                           float pf, bool lj, float& arvmu) {
    const MixedF& M = P.mf;
    const ReuseF& U = P.rf;
    const float rs = inv_distance(d2);
    const float s = cubic_s(U, d2 * rs * M.inv_h, rs);
    float vr = (vi.x - vj.x) * d.x + (vi.y - vj.y) * d.y;
    if (DIM == 3) vr += (vi.z - vj.z) * d.z;
    // approaching pairs only (vr < 0), evaluated by every lane and clamped
    const float rhos = vi.w + vj.w;
    const float w = fminf(vr, 0.0f) * rcp_approx((d2 + M.etq_h2) * rhos);
    if (MU || U.bulk != 0.0f) {
        const float mu = M.h * w * rhos;
        if (MU) arvmu = fmaxf(arvmu, -mu);
        pf = fmaf(U.bulk * mu, w, pf);
    }
    float m = s * fmaf(U.visc, w, pf);
    if (lj && d2 < U.lj_r2 && d2 > 0.0f) {
        const float rn = M.lj_rr0 * rs;
        const float rn2 = rn * rn, rn4 = rn2 * rn2, rn8 = rn4 * rn4;
        m -= U.lj_D * (rn8 * rn4 - rn4) * (rs * rs);
    }
    return m;
}

// update_acceleration over this step's neighbours: the list the density pass wrote
// (or the stencil search, where a searched particle may have
// more neighbours than a list holds: WV == 0). In 2D a neighbour's pressure comes
// with its velocity and density (V4.z); in 3D from PR. STD: the common method set
// (pair_coef), fixed at compile time. At most 64 registers (4 blocks of 256
// threads per SM): the gather hides its L1/L2 latency with warps.
// WV != 0: the whole step follows in the same thread (whole_particle with
// variant WV, thread 0 advancing the scalars into next): it reads nothing that
// another thread's whole step writes, because this step's copies (pos, V4, VD4)
// are not the ones the key pass writes (posn, V4n, VD4n), and the neighbours of
// every particle are listed (the density pass wrote those of searched particles
// too, which needs at most Vl<DIM>::cap neighbours per particle).
__device__ __forceinline__ void fetch_l1(const void* p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }
// The rows whole_particle and its key pass read of particle id.
template <int DIM>
__device__ __forceinline__ void fetch_whole(const State& S, uint32_t id) {
    fetch_l1(S.rx + id);
    fetch_l1(S.ry + id);
    fetch_l1(S.vx + id);
    fetch_l1(S.vy + id);
    if (DIM == 3) {
        fetch_l1(S.rz + id);
        fetch_l1(S.vz + id);
        fetch_l1(S.bfix4 + id);
    } else {
        fetch_l1(S.bfix2 + id);
        fetch_l1(S.bcxy + id);
    }
    fetch_l1(S.itype + id);
    fetch_l1(S.key_of + id);
    fetch_l1(S.slot + id);
}
template <int DIM, int SKF, bool STD, int WV, int L>
__global__ void __launch_bounds__(L > 1 ? 32 * L : kMaxGatherThreads, 4) k_forces_verlet(DevParams P, State S, Sorted G,
                                                                    StepScalars* __restrict__ scal,
                                                                    StepScalars* __restrict__ next,
                                                                    uint32_t* __restrict__ flags) {
    constexpr int B = kVlForceBatch<DIM, STD>;
    constexpr bool MU = WV == 0 || (WV & kVarRare) != 0;
    const uint32_t lane = threadIdx.x & 31u, sub = L > 1 ? threadIdx.x >> 5 : 0u;
    uint32_t k = L > 1 ? blockIdx.x * 32u + lane : blockIdx.x * blockDim.x + threadIdx.x;
    const bool active = k < P.n;
    // the warps of a split block meet below: its lanes past the end redo the last particle
    if (L > 1) k = min(k, P.n - 1u);
    double amag = 0, arvmu_d = 0;
    // launched while the density gather finishes: wait for it and its writes; the
    // split gather first fetches what that does not write (this particle's rows of
    // the whole step, into L1)
    if (WV != 0 && L > 1 && sub == 0) fetch_whole<DIM>(S, G.id[k]);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (L > 1 || active) {
        const ReuseF& U = P.rf;
        const uint32_t id = G.id[k];
        const Pos pj = G.pos[k];
        const bool fluid = pj.fluid();
        ForceAcc<DIM, SKF> F{P, G, G.V4[k], G.PR[k], 0.0f, false, false, false, false, false, 0, 0,
                             0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
        F.rhoj = F.vj.w;
        F.ext = P.repulsive && fluid;
        F.intf = true;
        F.visc = P.art_visc;
        F.avel = P.avg_vel;
        F.form1 = P.intf_form == 1;
        F.intf_skf = SKF ? SKF : P.intf_skf;
        F.av_skf = SKF ? SKF : P.av_skf;
        Kahan ax{0, 0}, ay{0, 0}, az{0, 0};
        Kahan avx{0, 0}, avy{0, 0}, avz{0, 0};
        // the general pair
        auto general = [&](const float4& vi, float2 pri, const Pos& pi, float3 d, float d2) {
            F.cax = F.cay = F.caz = F.cvx = F.cvy = F.cvz = 0.0f;
            F.pair_with(vi, pri, d.x, d.y, d.z, d2, pi.boundary() ? -1 : (pi.fluid() ? 1 : 0));
            ax.add(F.cax);
            ay.add(F.cay);
            if (DIM == 3) az.add(F.caz);
            if (F.avel) {
                avx.add(F.cvx);
                avy.add(F.cvy);
                if (DIM == 3) avz.add(F.cvz);
            }
        };
        auto one = [&](const float4& vi, float2 pr3, const Pos& pi) {
            const float3 d = separation<DIM>(pi, pj, U.u);
            const float d2 = distance2<DIM>(d, 0.0f);
            if (STD) {
                const float m = pair_coef<DIM, MU>(P, d, d2, F.vj, vi, (DIM == 3 ? pr3.y : vi.z) + F.prj.y,
                                                   F.ext && pi.boundary(), F.arvmu);
                // each pair's terms are added with compensation
                ax.add(d.x * m);
                ay.add(d.y * m);
                if (DIM == 3) az.add(d.z * m);
            } else if (DIM == 3) {
                general(vi, pr3, pi, d, d2);
            } else {  // p (form 1) or p/rho^2, as the density pass wrote it
                const float z = vi.z;
                general(vi, F.form1 ? make_float2(z, z * __frcp_rn(vi.w * vi.w)) : make_float2(z, z), pi, d, d2);
            }
        };
        if (!pj.absent()) {
            if (WV != 0 || G.vcount[k] != kListOver) {
                // four list words per load (the lanes of a warp load neighbouring uint4s), the
                // data of B of them together
                const uint32_t nc = sub_count<L>(G.ncount[k], sub);
                const uint4* const slab = reinterpret_cast<const uint4*>(G.nlist) + (size_t)sub * P.n + k;
                // (streaming, as in the density pass; the next words ahead of this group's data)
                uint4 ahead = make_uint4(0u, 0u, 0u, 0u);
                if (nc) ahead = __ldcs(slab);
                for (uint32_t e0 = 0; e0 < nc; e0 += 4) {
                    const uint4 w = ahead;
                    if (e0 + 4 < nc) ahead = __ldcs(slab + (size_t)(L * ((e0 >> 2) + 1)) * P.n);
                    const uint32_t en[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                    for (int h = 0; h < 4; h += B) {
                        Pos pb[B];
                        float4 vb[B];
                        float2 rb[B];
#pragma unroll
                        for (int j = 0; j < B; j++) {
                            if (e0 + h + j >= nc) continue;
                            pb[j] = G.pos[en[h + j]];
                            vb[j] = G.V4[en[h + j]];
                            if (DIM == 3) rb[j] = G.PR[en[h + j]];
                        }
#pragma unroll
                        for (int j = 0; j < B; j++) {
                            if (e0 + h + j >= nc) continue;
                            one(vb[j], DIM == 3 ? rb[j] : make_float2(0.0f, 0.0f), pb[j]);
                        }
                    }
                }
            } else if (sub == 0) {
                constexpr int NC = DIM == 3 ? 27 : 9;
                const Stencil<DIM> st(P, G.key[k]);
#pragma unroll 1
                for (int c = 0; c < NC; c++) {
                    uint32_t cell;
                    int sx, sy, sz;
                    if (!st.cell(c, cell, sx, sy, sz)) continue;
                    const uint32_t s = G.cell_start[cell];
                    if (s == kEmpty) continue;
                    const uint32_t e = G.cell_end[cell];
                    const bool wraps = wrapped<DIM>(sx, sy, sz);
#pragma unroll 1
                    for (uint32_t i = s; i < e; i++) {
                        if (i == k) continue;
                        const Pos pi = G.pos[i];
                        if (!searched_pair<DIM>(P, S, G, i, k, pi, pj, wraps)) continue;
                        one(G.V4[i], G.PR[i], pi);
                    }
                }
            }
        }
        if (L > 1) {  // the other warps' sums, then the first warp goes on alone
            constexpr int Q = (DIM == 3 ? 3 : 2) * (STD ? 1 : 2);
            __shared__ float part[L - 1 ? L - 1 : 1][2 * Q + 1][32];
            auto each = [&](auto&& f) {
                f(0, ax);
                f(1, ay);
                if (DIM == 3) f(2, az);
                if (!STD) {
                    f(DIM, avx);
                    f(DIM + 1, avy);
                    if (DIM == 3) f(5, avz);
                }
            };
            if (sub != 0) {
                each([&](int q, const Kahan& a) {
                    part[sub - 1][2 * q][lane] = a.s;
                    part[sub - 1][2 * q + 1][lane] = a.c;
                });
                part[sub - 1][2 * Q][lane] = F.arvmu;
            }
            __syncthreads();
            if (sub != 0) return;
#pragma unroll
            for (int u = 0; u < L - 1; u++) {
                each([&](int q, Kahan& a) {
                    a.add(part[u][2 * q][lane]);
                    a.c += part[u][2 * q + 1][lane];
                });
                F.arvmu = fmaxf(F.arvmu, part[u][2 * Q][lane]);
            }
        }
        if (L == 1 || active) {
            const F2 f = STD ? U.a : F2{1.0f, 0.0f};
            const double axd = value(scaled(ax, f)), ayd = value(scaled(ay, f)) - P.g;  // gravity along y (ExtForce.h), 2D and 3D
            const double azd = DIM == 3 ? value(scaled(az, f)) : 0.0;
            S.ax[id] = axd;
            S.ay[id] = ayd;
            if (DIM == 3) S.az[id] = azd;
            if (F.avel) {
                S.avx[id] = avx.value();
                S.avy[id] = avy.value();
                if (DIM == 3) S.avz[id] = avz.value();
            }
            arvmu_d = F.arvmu;
            if (P.dt_reduce) amag = sqrt(axd * axd + ayd * ayd + azd * azd);
            if (WV != 0) {
                const double dt = step_dt<(WV & kVarRare) != 0>(P, scal, flags, k == 0);
                if (k == 0) advance_scalars(P, scal, next, dt);
                whole_particle<DIM, WV>(P, S, G, id, dt, scal, flags, 1, L > 1, axd, ayd, azd);
            }
        }
    }
    if (P.dt_method == 2 && P.dt_reduce) {
        warp_max_bits(&scal->amax_bits, amag);
        warp_max_bits(&scal->mumax_bits, arvmu_d);
    }
}

}  // namespace

void launch_verlet_decide(cudaGraphConditionalHandle h, const uint32_t* rebuild, cudaStream_t st) {
    k_vl_decide<<<1, 1, 0, st>>>(h, rebuild);
}
void launch_verlet_reset(uint32_t* rebuild, uint32_t* gone, uint32_t* far, unsigned long long* builds,
                         cudaStream_t st) {
    k_vl_reset<<<1, 1, 0, st>>>(rebuild, gone, far, builds);
}
void launch_verlet_upload_check(uint32_t* rebuild, const uint32_t* gone, cudaStream_t st) {
    k_vl_upload_check<<<1, 1, 0, st>>>(rebuild, gone);
}
template <int DIM>
void launch_verlet_build(const DevParams& P, const State& S, const Sorted& G, cudaStream_t st) {
    if (P.reuse == kReuseCell) return launch_verlet_build_cell(P, S, G, st);
    k_vl_build<DIM><<<(P.n + kVlBuildThreads - 1) / kVlBuildThreads, kVlBuildThreads, 0, st>>>(P, S, G);
}
// Warps per 32 particles of the two gathers (DevParams::vl_split, fixed when a
// solver is created): four where a thread per particle leaves the SMs a few warps
// each, else one. us per step with 1 / 4 (8 is no faster; in 2D four is
// kernels_reuse_cell.cu): 2D, 6k particles 27.9 / 23.1, 22k 28.4 / 25.5, 34k 30.1 /
// 31.9, 43k 31.0 / 33.9, 66k 33.7 / 43.8; 3D, 67k 82.5 / 73.8, 139k 126.2 / 127.4,
// 240k 204 / 216. (A block keeps the registers of the warps that are done while its
// first warp finishes the step. The lines were drawn on earlier forms of both; the 2D
// one would lie at about 30,000 today, but results differ by rounding across it.)
int verlet_split(int dim, uint32_t n) { return n <= (dim == 3 ? 128000u : 36000u) ? 4 : 1; }

template <int DIM>
void launch_density_verlet(const DevParams& P, const State& S, const Sorted& G, StepScalars* scal, uint32_t* flags,
                           cudaStream_t st, int threads) {
    if (P.reuse == kReuseCell) return launch_density_cell(P, S, G, scal, flags, st);
    const bool cont = P.density_treatment != 0;
    const unsigned extra = has_pistons(P, S) ? 1 : 0;
#define RRSPH_DV(SKF, CONT)                                                                                           \
    do {                                                                                                              \
        if (DIM == 3 && P.vl_split == 4)                                                                              \
            k_density_verlet<DIM, SKF, CONT, DIM == 3 ? 4 : 1><<<(P.n + 31) / 32 + extra, 128, 128 * 32, st>>>(P, S, G, scal, flags);       \
        else                                                                                                          \
            k_density_verlet<DIM, SKF, CONT, 1><<<(P.n + threads - 1) / threads, threads, threads * 32, st>>>(P, S, G, scal, flags); \
    } while (0)
    if (P.all_cubic) {
        if (cont) RRSPH_DV(1, true);
        else RRSPH_DV(1, false);
    } else {
        if (cont) RRSPH_DV(0, true);
        else RRSPH_DV(0, false);
    }
#undef RRSPH_DV
}
template <int DIM>
void launch_forces_verlet(const DevParams& P, const State& S, const Sorted& G, StepScalars* scal,
                          StepScalars* scal_next, uint32_t* flags, cudaStream_t st, int threads, int whole) {
    const bool std_terms = P.all_cubic && P.intf_form != 1 && P.art_visc && !P.art_pressure && !P.avg_vel;
    const int wv = whole ? (kVarMixed | (P.density_treatment != 0 ? kVarCont : 0) |
                            (P.avg_vel || P.dt_method == 2 ? kVarRare : 0))
                         : 0;
    if (P.reuse == kReuseCell) return launch_forces_cell(P, S, G, scal, scal_next, flags, st, std_terms, wv);
// the force gather follows the density gather with a programmatic dependency:
// its blocks launch as the density gather's last blocks run, then wait for it
#define RRSPH_FV(SKF, STD, WV)                                                                                       \
    do {                                                                                                             \
        if (DIM == 3 && P.vl_split == 4)                                                                             \
            launch_after(k_forces_verlet<DIM, SKF, STD, WV, DIM == 3 ? 4 : 1>, (P.n + 31) / 32, 128, st, P, S, G, scal, scal_next, flags); \
        else                                                                                                         \
            launch_after(k_forces_verlet<DIM, SKF, STD, WV, 1>, (P.n + threads - 1) / threads, threads, st, P, S, G, \
                         scal, scal_next, flags);                                                                    \
    } while (0)
#define RRSPH_FV_WV(SKF, STD)                                                          \
    do {                                                                               \
        switch (wv) {                                                                  \
        case 0: RRSPH_FV(SKF, STD, 0); break;                                          \
        case kVarMixed: RRSPH_FV(SKF, STD, kVarMixed); break;                          \
        case kVarMixed | kVarCont: RRSPH_FV(SKF, STD, kVarMixed | kVarCont); break;    \
        case kVarMixed | kVarRare: RRSPH_FV(SKF, STD, kVarMixed | kVarRare); break;    \
        default: RRSPH_FV(SKF, STD, kVarMixed | kVarCont | kVarRare);                  \
        }                                                                              \
    } while (0)
    if (std_terms) RRSPH_FV_WV(1, true);
    else if (P.all_cubic) RRSPH_FV_WV(1, false);
    else RRSPH_FV_WV(0, false);
#undef RRSPH_FV_WV
#undef RRSPH_FV
}

namespace {

// The neighbour list the last density pass of the reuse step wrote, as particle
// ids: row G.id[k] of `list` gets the ids of slot k's.
template <int DIM, int L>
__global__ void k_nlist_export(DevParams P, Sorted G, uint32_t* __restrict__ counts, uint32_t* __restrict__ list,
                               uint32_t max_per, uint32_t* __restrict__ flags) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= P.n) return;
    const uint32_t id = G.id[k];
    const uint32_t index = P.reuse == kReuseCell ? kCellEntryIndex : 0xFFFFFFFFu;
    uint32_t c = 0;
    for (uint32_t u = 0; u < (uint32_t)L; u++) {
        const uint32_t m = sub_count<L>(G.ncount[k], u);
        for (uint32_t e = 0; e < m; e++, c++)
            if (c < max_per)
                list[(size_t)id * max_per + c] =
                    G.id[G.nlist[((size_t)(u + L * (e >> 2)) * P.n + k) * 4 + (e & 3u)] & index];
    }
    counts[id] = c;
    // a searched particle stores at most the list capacity: a full row may have
    // lost entries, which this copy cannot show
    const bool clipped = c == (uint32_t)Vl<DIM>::cap && G.vcount[k] == kListOver;
    if (c > max_per || clipped) atomicOr(flags, RRSPH_FLAG_NEIGHBOUR_OVERFLOW);
}

}  // namespace

template <int DIM>
void launch_nlist_export(const DevParams& P, const Sorted& G, uint32_t* counts, uint32_t* list, uint32_t max_per,
                         uint32_t* flags, cudaStream_t st) {
    const unsigned blocks = (P.n + 255) / 256;
    if (P.vl_split == 4) k_nlist_export<DIM, 4><<<blocks, 256, 0, st>>>(P, G, counts, list, max_per, flags);
    else k_nlist_export<DIM, 1><<<blocks, 256, 0, st>>>(P, G, counts, list, max_per, flags);
}

namespace {
__global__ void k_clear_cells(uint32_t* __restrict__ cell_start, uint32_t max_cells) {
    const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c < max_cells) cell_start[c] = kEmpty;
}
}  // namespace

void launch_clear_cells(uint32_t* cell_start, uint32_t max_cells, cudaStream_t st) {
    k_clear_cells<<<(max_cells + 255) / 256, 256, 0, st>>>(cell_start, max_cells);
}

template void launch_nlist_export<2>(const DevParams&, const Sorted&, uint32_t*, uint32_t*, uint32_t, uint32_t*,
                                     cudaStream_t);
template void launch_nlist_export<3>(const DevParams&, const Sorted&, uint32_t*, uint32_t*, uint32_t, uint32_t*,
                                     cudaStream_t);

template void launch_verlet_build<2>(const DevParams&, const State&, const Sorted&, cudaStream_t);
template void launch_verlet_build<3>(const DevParams&, const State&, const Sorted&, cudaStream_t);
template void launch_density_verlet<2>(const DevParams&, const State&, const Sorted&, StepScalars*, uint32_t*,
                                       cudaStream_t, int);
template void launch_density_verlet<3>(const DevParams&, const State&, const Sorted&, StepScalars*, uint32_t*,
                                       cudaStream_t, int);
template void launch_forces_verlet<2>(const DevParams&, const State&, const Sorted&, StepScalars*, StepScalars*,
                                      uint32_t*, cudaStream_t, int, int);
template void launch_forces_verlet<3>(const DevParams&, const State&, const Sorted&, StepScalars*, StepScalars*,
                                      uint32_t*, cudaStream_t, int, int);

}  // namespace rrsph
