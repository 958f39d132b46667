// kernels_reuse_cell.cu — the FP32-mixed step with neighbour reuse in 2D for few
// particles (the split gathers): kernels_reuse.cu's scheme on cell-relative float
// positions, each list entry with its cell offset as a code. Fixed-point positions
// give these sizes no speed, which latency bounds (6k dam break 24.6 us a step with
// them, 24.1 without, 2.5k tank 24.6 both), and would move their results (r by 3.5e-9
// over 50 steps of the 6k dam break, which runs long between two layers), though fixed
// point is the more exact of the two (density 3.5e-8 against 4.8e-8 off FP64).
#include "reuse.cuh"

namespace rrsph {

namespace {

constexpr uint32_t kVlNone = 0xFFFFFFFFu;  // padding of a list row (never an entry)
constexpr int kVlBatch = 4;       // list entries the density gather loads together (one uint4)
// neighbours the force gather loads together: four for the 2D common method
// set, two elsewhere (four would spill the registers of the general pair)
template <bool STD>
constexpr int kVlForceBatch = STD ? 4 : 2;
constexpr int kWarps = 4;  // warps per 32 particles

// List entry = sorted index | cell code << Vl::shift, with the code of
// the candidate's cell offset (dx, dy) in [-2, 2]^2: (dx + 2) * 5 + (dy + 2).
struct Vl {
    static constexpr int cap = kVerletCap2;
    static constexpr int shift = 27;
    static constexpr uint32_t index = (1u << shift) - 1u;
    static constexpr uint32_t cmax = kMaxCellCoord2;  // largest cell coordinate of a key
};

__device__ __forceinline__ uint32_t vl_code(int dx, int dy) {
    return (uint32_t)((dx + 2) * 5 + (dy + 2)) << Vl::shift;
}
// The offset of an entry's code, shifted by +2 per axis (0..4).
__device__ __forceinline__ void vl_offset(uint32_t en, uint32_t& cx, uint32_t& cy) {
    const uint32_t c = en >> Vl::shift;
    cx = (c * 13u) >> 6;  // c / 5, exact for c < 32
    cy = c - 5u * cx;
}

// The cubic W(q) of kernel_wf as selects: every lane runs the same instructions.
__device__ __forceinline__ float cubic_wf_sel(float f, float q) {
    const float t = 2.0f - q;
    const float w1 = f * ((2.0f / 3.0f - q * q) + q * q * q * 0.5f);
    const float w2 = f * ((1.0f / 6.0f) * (t * t * t));
    return q <= 1.0f ? w1 : (q <= 2.0f ? w2 : 0.0f);
}

// The window of cell offsets along one axis a particle at offset p from its
// cell's lower edge searches: the cell equals the cutoff and the skin is at
// most h, so a candidate within cutoff + skin lies at most two cells away, and
// two only on the side whose edge is within one skin.
__device__ __forceinline__ void vl_window(float p, uint32_t c, float cell, float edge, int& lo, int& hi) {
    lo = (p < edge && c >= 2) ? -2 : (c >= 1 ? -1 : 0);
    hi = (p > cell - edge && c + 2 <= Vl::cmax) ? 2 : (c + 1 <= Vl::cmax ? 1 : 0);
}

// Distance along one axis from a particle at offset p in [0, cell] from its
// cell's lower edge to the nearest side of the cell d cells away.
__device__ __forceinline__ float gap_to_cell(int d, float p, float cell) {
    return d > 0 ? (float)d * cell - p : (d < 0 ? p - (float)(d + 1) * cell : 0.0f);
}

// After this step's grid (sort + reorder): each particle's candidates in groups of
// four (the lanes of a warp store neighbouring uint4s), in cell order x outer, the
// last group padded. A block takes 32 particles and a warp the cells of one x of
// their windows, its ranges of particles first and then these in one loop; the
// four warps' entries, kept in shared memory, make up the list in order (one
// thread a particle walked the cells one by one, a chain of dependent loads on a
// nearly empty chip: 26 us a rebuild of 6k
// particles, 9.8 so, the 6k dam break 23.7 -> 22.1 us a step).
__global__ void __launch_bounds__(32 * kWarps) k_vl_build(DevParams P, State S, Sorted G) {
    constexpr uint32_t CAP = Vl::cap;
    __shared__ uint32_t entries[kWarps][CAP][32];
    __shared__ uint2 ranges[5][32 * kWarps];  // a cell's first particle; its end | dy + 2 << Vl::shift
    __shared__ uint32_t counts[kWarps][32];
    const uint32_t lane = threadIdx.x & 31u, sub = threadIdx.x >> 5, t = threadIdx.x;
    const uint32_t k = blockIdx.x * 32u + lane;
    const bool active = k < P.n;
    const MixedF& M = P.mf;
    uint32_t nl = 0;
    if (active) {
        const uint32_t key = G.key[k];
        const float4 pj = G.P4[k];
        const uint32_t cx = second_bits(key), cy = second_bits(key >> 1);
        const bool absent = __float_as_int(pj.w) == P.type_non_existent;
        if (sub == 0) {
            const uint32_t id = G.id[k];
            S.bcxy[id] = cx | (cy << 16);
            S.boff[id] = make_float2(pj.x, pj.y);
            S.slot[id] = k;
            if (absent) atomicOr(S.vl_gone, 1u);
        }
        if (!absent) {
            int x0, x1, y0, y1;
            vl_window(pj.x, cx, M.cell, P.vl_skin_edge, x0, x1);
            vl_window(pj.y, cy, M.cell, P.vl_skin_edge, y0, y1);
            // (a window is five cells wide only where the skin is h, in the cell's middle)
            const int last = sub == kWarps - 1 ? x1 : min(x1, x0 + (int)sub);
            for (int dx = x0 + (int)sub; dx <= last; dx++) {
                const uint32_t mx = split2_32(cx + dx);
                const float gx = gap_to_cell(dx, pj.x, M.cell);
                uint32_t nr = 0;
#pragma unroll
                for (int j = 0; j < 5; j++) {
                    const int dy = y0 + j;
                    // a cell none of whose points lies within the list cutoff of the
                    // particle holds no candidate: the distance from the particle to the
                    // cell's nearest side, per axis
                    const float gy = gap_to_cell(dy, pj.y, M.cell);
                    const uint32_t c = mx | (split2_32(cy + dy) << 1);
                    if (dy <= y1 && !(gx * gx + gy * gy >= P.vl_cut2) && c < P.max_cells) {
                        const uint32_t s = G.cell_start[c], e = G.cell_end[c];
                        if (s != kEmpty) ranges[nr++][t] = make_uint2(s, e | ((uint32_t)(dy + 2) << Vl::shift));
                    }
                }
                const float shx = (float)dx * M.cell - pj.x;
                for (uint32_t q = 0; q < nr; q++) {
                    const uint2 se = ranges[q][t];
                    const uint32_t e = se.y & Vl::index;
                    const int dy = (int)(se.y >> Vl::shift) - 2;
                    const float shy = (float)dy * M.cell - pj.y;
                    const uint32_t code = vl_code(dx, dy);
                    // four at a time: their loads issue together (an index past the cell's
                    // end loads its last particle and is skipped)
                    for (uint32_t i0 = se.x; i0 < e; i0 += kVlBatch) {
                        float4 p[kVlBatch];
#pragma unroll
                        for (int u = 0; u < kVlBatch; u++) p[u] = G.P4[min(i0 + u, e - 1u)];
#pragma unroll
                        for (int u = 0; u < kVlBatch; u++) {
                            const uint32_t i = i0 + u;
                            const float ddx = p[u].x + shx, ddy = p[u].y + shy;
                            // past the cell's end, itself, or non-existent (stays so): no candidate
                            const bool in = ddx * ddx + ddy * ddy < P.vl_cut2 && i < e && i != k &&
                                            __float_as_int(p[u].w) != P.type_non_existent;
                            if (in && nl < CAP) entries[sub][nl][lane] = i | code;
                            nl += in;
                        }
                    }
                }
            }
        }
    }
    counts[sub][lane] = nl;
    __syncthreads();
    if (!active) return;
    uint32_t end[kWarps];  // of each warp's entries in the list
    uint32_t total = 0;
#pragma unroll
    for (uint32_t u = 0; u < kWarps; u++) end[u] = total += counts[u][lane];
    const uint32_t listed = min(total, CAP);
    for (uint32_t g = sub; 4 * g < listed; g += kWarps) {
        uint32_t w[4];
#pragma unroll
        for (uint32_t j = 0; j < 4; j++) {
            const uint32_t e = 4 * g + j;
            const uint32_t u = (e >= end[0]) + (e >= end[1]) + (e >= end[2]);
            const uint32_t before = u == 0 ? 0u : (u == 1 ? end[0] : (u == 2 ? end[1] : end[2]));
            w[j] = e < listed ? entries[u][e - before][lane] : kVlNone;
        }
        reinterpret_cast<uint4*>(G.vlist)[(size_t)g * P.n + k] = make_uint4(w[0], w[1], w[2], w[3]);
    }
    if (sub != 0) return;
    G.vcount[k] = total <= CAP ? total : kListOver;
    if (total > CAP) {  // its search needs a fresh grid each step
        atomicOr(S.vl_rebuild, 1u);
        atomicOr(S.vl_gone, 2u);
    }
}

// The split gathers: a block of four warps takes 32 particles, warp `sub` their
// list groups sub, sub + 4, ..., and the first warp adds the partial sums up and
// goes on alone. With few particles a thread walking its whole list is one long
// chain of dependent loads on a nearly empty chip. A warp's neighbours go to the
// slab groups it reads (sub + 4 j), so no warp waits for another's count; the
// four counts share the particle's word.
__device__ __forceinline__ uint32_t sub_count(uint32_t word, uint32_t sub) { return (word >> (sub * 8)) & 0xFFu; }
// Slab offset of neighbour e of warp `sub` (in words, from the particle's uint4).
__device__ __forceinline__ size_t slab_at(uint32_t n, uint32_t sub, uint32_t e) {
    return (size_t)(sub + kWarps * (e >> 2)) * 4 * n + (e & 3u);
}
// Neighbour e of a list in consecutive groups, and the word of one of c entries.
__device__ __forceinline__ size_t list_at(uint32_t n, uint32_t e) { return (size_t)(e >> 2) * 4 * n + (e & 3u); }
__device__ __forceinline__ uint32_t packed_counts(uint32_t c) {
    uint32_t word = 0;
    for (uint32_t g = 0; 4 * g < c; g++) word += min(4u, c - 4 * g) << ((g % kWarps) * 8);
    return word;
}

// One candidate's contribution to the density gather: W (summation) or the
// continuity rate with its delta-SPH term (density_con, Density.h:63-114,
// the same arithmetic as k_density_mixed).
template <int SKF, bool CONT>
__device__ __forceinline__ float density_term(const MixedF& M, int skf, float f, float dx, float dy, float d2,
                                              float4 vdi, float4 vdj, bool delta) {
    const float inv_dist = inv_distance(d2);
    const float q = d2 * inv_dist * M.inv_h;
    if (!CONT) return SKF == 1 ? cubic_wf_sel(f, q) : kernel_wf(skf, f, q);
    const float sc = SKF == 1 ? cubic_dwdr_sel(f, q, inv_dist, M.inv_h)
                              : kernel_dwdr_scalef(skf, f, q, inv_dist, M.inv_h);
    float vcc = (vdi.x - vdj.x) * dx + (vdi.y - vdj.y) * dy;
    float term = vcc * sc;
    if (delta) {
        const float rho_factor = __fdividef(vd4_drho<2>(vdi, vdj), M.rho0 + vdi.w);
        term += 2.0f * M.dhc * (rho_factor * -sc);
    }
    return term;
}

// density_sum (Density.h:25-61) + EOS, or density_con (Density.h:63-114), over
// the candidate list: the entries within the cutoff are this step's
// neighbours, written to nlist for the force pass. A particle whose list
// overflowed searches the stencil cells (the grid is rebuilt every step while
// one does) and writes its neighbours too.
template <int SKF, bool CONT>
__global__ void __launch_bounds__(32 * kWarps) k_density_verlet(DevParams P, State S, Sorted G,
                                                                     StepScalars* __restrict__ scal,
                                                                     uint32_t* __restrict__ flags) {
    constexpr int CAP = Vl::cap;
    constexpr uint32_t IDX = Vl::index;
    // the force gather may launch now: it waits for this grid at its start (griddepcontrol.wait)
    asm volatile("griddepcontrol.launch_dependents;");
    if (blockIdx.x * 32u >= P.n) {  // the extra block
        piston_block(P, S, scal);
        return;
    }
    const uint32_t lane = threadIdx.x & 31u, sub = threadIdx.x >> 5;
    const uint32_t k = blockIdx.x * 32u + lane;
    const bool active = k < P.n;
    uint32_t cnt = 0, word = 0;
    Kahan acc{0.0f, 0.0f};
    if (active) {
        const MixedF& M = P.mf;
        const float4 pj = G.P4[k];
        const int32_t tj = __float_as_int(pj.w);
        const int skf = SKF ? SKF : P.density_skf;
        const float f = M.kf[skf];
        const bool delta = CONT && P.density_treatment == 2;
        const float4 vdj = CONT ? G.VD4[k] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        uint32_t* const nslab = G.nlist + (size_t)k * 4;  // neighbour e at nslab[slab_at(e)]
        if (tj != P.type_non_existent) {
            const uint32_t vc = G.vcount[k];
            if (vc != kListOver) {
                const uint4* slab = reinterpret_cast<const uint4*>(G.vlist) + k;  // group g at slab[g * n]
                // shift of offset code (cx, cy) = (cx - 2, cy - 2) cells, relative to this particle
                const float bx = -2.0f * M.cell - pj.x, by = -2.0f * M.cell - pj.y;
                // groups of four entries (one load, the next group's issued before this
                // one's particles are loaded), then their particles, loaded together;
                // the body has no branch but the rare guard-band test, and each group's
                // sum is added with compensation
                // (list words are read once a step: streaming loads keep L1 for the neighbours' data)
                uint4 w = 4 * sub < vc ? __ldcs(slab + (size_t)sub * P.n)
                                       : make_uint4(kVlNone, kVlNone, kVlNone, kVlNone);
                for (uint32_t e0 = 4 * sub; e0 < vc; e0 += kVlBatch * kWarps) {
                    const uint4 wn = e0 + kVlBatch * kWarps < vc ? __ldcs(slab + (size_t)((e0 >> 2) + kWarps) * P.n) : w;
                    const uint32_t en[kVlBatch] = {w.x, w.y, w.z, w.w};
                    float4 pb[kVlBatch];
#pragma unroll
                    for (int j = 0; j < kVlBatch; j++)
                        pb[j] = en[j] != kVlNone ? G.P4[en[j] & IDX] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    float part = 0.0f;
#pragma unroll
                    for (int j = 0; j < kVlBatch; j++) {
                        uint32_t cx, cy;
                        vl_offset(en[j], cx, cy);
                        const float dx = pb[j].x + fmaf((float)cx, M.cell, bx);
                        const float dy = pb[j].y + fmaf((float)cy, M.cell, by);
                        const float d2 = dx * dx + dy * dy;
                        bool in = en[j] != kVlNone && __float_as_int(pb[j].w) != P.type_non_existent &&
                                  d2 < M.cut2_hi;
                        if (in && !(d2 < M.cut2_lo)) in = within_cutoff<2>(P, S, G, en[j] & IDX, k, d2);
                        const float4 vdi = CONT && in ? G.VD4[en[j] & IDX] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                        const float t = density_term<SKF, CONT>(M, skf, f, dx, dy, d2, vdi, vdj, delta);
                        part += in ? t : 0.0f;
                        if (in) nslab[slab_at(P.n, sub, cnt)] = en[j];
                        cnt += in;
                    }
                    acc.add(M.mass * part);
                    w = wn;
                }
                word = cnt;
            } else if (sub == 0) {
                const Stencil<2> st(P, G.key[k]);
#pragma unroll 1
                for (int c = 0; c < 9; c++) {
                    uint32_t cell;
                    int sx, sy, sz;
                    if (!st.cell(c, cell, sx, sy, sz)) continue;
                    const uint32_t s = G.cell_start[cell];
                    if (s == kEmpty) continue;
                    const uint32_t e = G.cell_end[cell];
                    const float shx = (float)sx * M.cell - pj.x;
                    const float shy = (float)sy * M.cell - pj.y;
                    float part = 0.0f;
                    for (uint32_t i = s; i < e; i++) {
                        if (i == k) continue;
                        const float4 pi = G.P4[i];
                        if (__float_as_int(pi.w) == P.type_non_existent) continue;
                        const float dx = pi.x + shx, dy = pi.y + shy;
                        const float d2 = dx * dx + dy * dy;
                        if (!within_cutoff<2>(P, S, G, i, k, d2)) continue;
                        // this step's neighbour list too (the grid is this step's: the stencil
                        // offsets are within one cell)
                        if (cnt < (uint32_t)CAP)
                            nslab[list_at(P.n, cnt)] = i | vl_code(sx, sy);
                        cnt++;
                        const float4 vdi = CONT ? G.VD4[i] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                        part += density_term<SKF, CONT>(M, skf, f, dx, dy, d2, vdi, vdj, delta);
                    }
                    acc.add(M.mass * part);
                }
                word = packed_counts(min(cnt, (uint32_t)CAP));
            }
        }
    }
    __shared__ float ps[kWarps][32], pc[kWarps][32];
    __shared__ uint32_t pn[kWarps][32];
    ps[sub][lane] = acc.s;
    pc[sub][lane] = acc.c;
    pn[sub][lane] = cnt;
    __syncthreads();
    if (sub != 0) return;
    if (active) {
        // (an over-full list was searched by this warp alone, its counts packed)
        const bool listed = G.vcount[k] != kListOver;
#pragma unroll
        for (int u = 1; u < kWarps; u++) {
            acc.add(ps[u][lane]);
            acc.c += pc[u][lane];
            cnt += pn[u][lane];
            if (listed) word |= pn[u][lane] << ((uint32_t)u * 8);
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
            const float d = ((acc.s - M.rho0_minus_w0_hi) - acc.c) - M.rho0_minus_w0_lo;
            const float rho = M.rho0 + d;
            const float pr = eos_pf(M, d);
            const float2 prr = make_float2(pr, pr * __frcp_rn(rho * rho));
            // V4.zw = (the pressure the force pass reads of a neighbour: p (form 1) or p/rho^2, rho)
            reinterpret_cast<float2*>(G.V4 + k)[1] = make_float2(P.intf_form == 1 ? prr.x : prr.y, rho);
            G.PR[k] = prr;
            S.rho[id] = P.rho0 + f2d(d);
            S.p[id] = f2d(pr);
        } else {
            const float d = (float)(S.rho[id] - P.rho0);
            const float pr = eos_pf(M, d);
            const float rf = G.V4[k].w;  // rho_predict, the density of the forces
            const float2 prr = make_float2(pr, pr * __frcp_rn(rf * rf));
            G.V4[k].z = P.intf_form == 1 ? prr.x : prr.y;
            G.PR[k] = prr;
            S.p[id] = pr;
            S.drho[id] = acc.value();
        }
    }
    warp_sum_add(&scal->pairs, cnt);
}

// update_acceleration over this step's neighbours: the list the density pass
// wrote (or the stencil search for an overflowed list). A neighbour's pressure
// comes with its velocity and density (V4.z). STD: the common method set of
// ForceAcc::pair_std, fixed at compile time.
// WV != 0: the whole step follows in the same thread (whole_particle with
// variant WV, thread 0 advancing the scalars into next): it reads nothing that
// another thread's whole step writes, because this step's copies (P4, V4, VD4)
// are not the ones the key pass writes (P4n, V4n, VD4n), and the list of every
// particle is complete (the density pass wrote the neighbours of overflowed
// lists too, which needs at most Vl::cap neighbours per particle).
__device__ __forceinline__ void fetch_l1(const void* p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }
// The rows whole_particle and its key pass read of particle id.
__device__ __forceinline__ void fetch_whole(const State& S, uint32_t id) {
    fetch_l1(S.rx + id);
    fetch_l1(S.ry + id);
    fetch_l1(S.vx + id);
    fetch_l1(S.vy + id);
    fetch_l1(S.boff + id);
    fetch_l1(S.itype + id);
    fetch_l1(S.key_of + id);
    fetch_l1(S.bcxy + id);
    fetch_l1(S.slot + id);
}
template <int SKF, bool STD, int WV>
__global__ void __launch_bounds__(32 * kWarps, 4) k_forces_verlet(DevParams P, State S, Sorted G,
                                                                    StepScalars* __restrict__ scal,
                                                                    StepScalars* __restrict__ next,
                                                                    uint32_t* __restrict__ flags) {
    constexpr uint32_t IDX = Vl::index;
    const uint32_t lane = threadIdx.x & 31u, sub = threadIdx.x >> 5;
    uint32_t k = blockIdx.x * 32u + lane;
    const bool active = k < P.n;
    // the warps of a block meet below: its lanes past the end redo the last particle
    k = min(k, P.n - 1u);
    double amag = 0, arvmu_d = 0;
    // launched while the density gather finishes: fetch what that does not write
    // (this particle's rows of the whole step, into L1), then wait for it and its writes
    if (WV != 0 && sub == 0) fetch_whole(S, G.id[k]);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const MixedF& M = P.mf;
    const uint32_t id = G.id[k];
    const float4 pj4 = G.P4[k];
    const int32_t tj = __float_as_int(pj4.w);
    ForceAcc<2, SKF> F{P, G, G.V4[k], G.PR[k], 0.0f, false, false, false, false, false, 0, 0,
                         0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    F.rhoj = F.vj.w;
    F.ext = P.repulsive && tj > 0;
    F.intf = true;
    F.visc = P.art_visc;
    F.avel = P.avg_vel;
    F.form1 = P.intf_form == 1;
    F.intf_skf = SKF ? SKF : P.intf_skf;
    F.av_skf = SKF ? SKF : P.av_skf;
    Kahan ax{0, 0}, ay{0, 0};
    Kahan avx{0, 0}, avy{0, 0};
    if (tj != P.type_non_existent) {
        const uint32_t vc = G.vcount[k];
        if (WV != 0 || vc != kListOver) {
            // this step's neighbours, four list words per load (the lanes of a
            // warp load neighbouring uint4s), their data two at a time
            const uint32_t nc = sub_count(G.ncount[k], sub);
            const uint4* nslab = reinterpret_cast<const uint4*>(G.nlist) + k;  // group g at nslab[g * n]
            const float bx = -2.0f * M.cell - pj4.x, by = -2.0f * M.cell - pj4.y;
            for (uint32_t e0 = 0; e0 < nc; e0 += 4) {
                // streaming, as in the density pass
                const uint4 w = __ldcs(nslab + (size_t)(sub + kWarps * (e0 >> 2)) * P.n);
                const uint32_t eg[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                for (int h = 0; h < 4; h += kVlForceBatch<STD>) {
                    uint32_t en[kVlForceBatch<STD>];
                    float4 pb[kVlForceBatch<STD>], vb[kVlForceBatch<STD>];
#pragma unroll
                    for (int j = 0; j < kVlForceBatch<STD>; j++) en[j] = e0 + h + j < nc ? eg[h + j] : kVlNone;
#pragma unroll
                    for (int j = 0; j < kVlForceBatch<STD>; j++) {
                        if (en[j] == kVlNone) continue;
                        const uint32_t i = en[j] & IDX;
                        pb[j] = G.P4[i];
                        vb[j] = G.V4[i];
                    }
                    // each pair's terms are added with compensation (no per-cell
                    // partial sums, whose flushes would split the warp)
#pragma unroll
                    for (int j = 0; j < kVlForceBatch<STD>; j++) {
                        if (en[j] == kVlNone) continue;
                        uint32_t cx, cy;
                        vl_offset(en[j], cx, cy);
                        const float dx = pb[j].x + fmaf((float)cx, M.cell, bx);
                        const float dy = pb[j].y + fmaf((float)cy, M.cell, by);
                        const float d2 = dx * dx + dy * dy;
                        F.cax = F.cay = F.caz = F.cvx = F.cvy = F.cvz = 0.0f;
                        if (STD) {
                            F.pair_std(vb[j], dx, dy, d2, __float_as_int(pb[j].w));
                        } else {  // p (form 1) or p/rho^2, as the density pass wrote it
                            const float z = vb[j].z;
                            const float2 pri = F.form1 ? make_float2(z, z * __frcp_rn(vb[j].w * vb[j].w)) : make_float2(z, z);
                            F.pair_with(vb[j], pri, dx, dy, 0.0f, d2, __float_as_int(pb[j].w));
                        }
                        ax.add(F.cax);
                        ay.add(F.cay);
                        if (!STD && F.avel) {
                            avx.add(F.cvx);
                            avy.add(F.cvy);
                        }
                    }
                }
            }
        } else if (sub == 0) {
            const Stencil<2> st(P, G.key[k]);
#pragma unroll 1
            for (int c = 0; c < 9; c++) {
                uint32_t cell;
                int sx, sy, sz;
                if (!st.cell(c, cell, sx, sy, sz)) continue;
                const uint32_t s = G.cell_start[cell];
                if (s == kEmpty) continue;
                const uint32_t e = G.cell_end[cell];
                const float shx = (float)sx * M.cell - pj4.x;
                const float shy = (float)sy * M.cell - pj4.y;
                F.cax = F.cay = F.caz = F.cvx = F.cvy = F.cvz = 0.0f;
                for (uint32_t i = s; i < e; i++) {
                    if (i == k) continue;
                    const float4 pi4 = G.P4[i];
                    const int32_t ti = __float_as_int(pi4.w);
                    if (ti == P.type_non_existent) continue;
                    const float dx = pi4.x + shx, dy = pi4.y + shy;
                    const float d2 = dx * dx + dy * dy;
                    if (!within_cutoff<2>(P, S, G, i, k, d2)) continue;
                    F.pair(i, dx, dy, 0.0f, d2, ti);
                }
                ax.add(F.cax);
                ay.add(F.cay);
                if (F.avel) {
                    avx.add(F.cvx);
                    avy.add(F.cvy);
                }
            }
        }
    }
    // the other warps' sums, then the first warp goes on alone
    constexpr int Q = STD ? 2 : 4;
    __shared__ float part[kWarps - 1][2 * Q + 1][32];
    auto each = [&](auto&& f) {
        f(0, ax);
        f(1, ay);
        if (!STD) {
            f(2, avx);
            f(3, avy);
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
    for (int u = 0; u < kWarps - 1; u++) {
        each([&](int q, Kahan& a) {
            a.add(part[u][2 * q][lane]);
            a.c += part[u][2 * q + 1][lane];
        });
        F.arvmu = fmaxf(F.arvmu, part[u][2 * Q][lane]);
    }
    if (active) {
        const double axd = ax.value(), ayd = ay.value() - P.g;
        S.ax[id] = axd;
        S.ay[id] = ayd;
        if (F.avel) {
            S.avx[id] = avx.value();
            S.avy[id] = avy.value();
        }
        arvmu_d = F.arvmu;
        if (P.dt_reduce) amag = sqrt(axd * axd + ayd * ayd);
        if (WV != 0) {
            const double dt = step_dt<(WV & kVarRare) != 0>(P, scal, flags, k == 0);
            if (k == 0) advance_scalars(P, scal, next, dt);
            whole_particle<2, WV>(P, S, G, id, dt, scal, flags, 1, true, axd, ayd, 0.0);
        }
    }
    if (P.dt_method == 2 && P.dt_reduce) {
        warp_max_bits(&scal->amax_bits, amag);
        warp_max_bits(&scal->mumax_bits, arvmu_d);
    }
}

}  // namespace

void launch_verlet_build_cell(const DevParams& P, const State& S, const Sorted& G, cudaStream_t st) {
    k_vl_build<<<(P.n + 31) / 32, 32 * kWarps, 0, st>>>(P, S, G);
}
void launch_density_cell(const DevParams& P, const State& S, const Sorted& G, StepScalars* scal, uint32_t* flags,
                         cudaStream_t st) {
    const unsigned blocks = (P.n + 31) / 32 + (has_pistons(P, S) ? 1 : 0);
    const bool cont = P.density_treatment != 0;
    if (P.all_cubic) {
        if (cont) k_density_verlet<1, true><<<blocks, 32 * kWarps, 0, st>>>(P, S, G, scal, flags);
        else k_density_verlet<1, false><<<blocks, 32 * kWarps, 0, st>>>(P, S, G, scal, flags);
    } else {
        if (cont) k_density_verlet<0, true><<<blocks, 32 * kWarps, 0, st>>>(P, S, G, scal, flags);
        else k_density_verlet<0, false><<<blocks, 32 * kWarps, 0, st>>>(P, S, G, scal, flags);
    }
}
void launch_forces_cell(const DevParams& P, const State& S, const Sorted& G, StepScalars* scal,
                        StepScalars* scal_next, uint32_t* flags, cudaStream_t st, bool std_terms, int wv) {
#define RRSPH_FV(SKF, STD, WV) \
    launch_after(k_forces_verlet<SKF, STD, WV>, (P.n + 31) / 32, 32 * kWarps, st, P, S, G, scal, scal_next, flags)
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

}  // namespace rrsph
