// kernels.cuh — device buffers of a solver and the launchers of its kernels.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "common.cuh"

namespace rrsph {

// Particle state in id order (the reference's arrays), double precision.
struct State {
    double *rx, *ry, *rz;      // positions
    double *vx, *vy, *vz;      // velocities
    double *ax, *ay, *az;      // accelerations of the last force evaluation
    double *avx, *avy, *avz;   // XSPH average velocity (average_velocity only)
    double *vpx, *vpy, *vpz;   // v_predict
    double *rho, *p, *drho, *rho_pred;
    double *mu;                // max |mu_ij| per particle (rrsph_forces only)
    int32_t* itype;
    uint32_t* key_of;          // cell key used by the last grid build, per id
    int32_t* wave_tank;        // piston of each particle in wave_law, -1 for none (null: the params' wave maker)
    const PistonLaw* wave_law; // wave-maker table
    double* wave_vx;           // its pistons' velocities of this step (piston_block)
    uint32_t wave_count;
    // FP32-mixed step only (null otherwise), written by the key pass, id order:
    float2* coff2;             // 2D: offset of r from its cell's lower edge
    float4* coff4;             // 3D: the same (x, y, z)
    float2* vpf2;              // 2D: v_predict in float
    float4* vpf4;              // 3D: the same (x, y, z)
    // mixed step with neighbour reuse (null otherwise), id order:
    int2* fix2;                // 2D: fixed-point position (Pos)
    int4* fix4;                // 3D: the same (x, y, z)
    int2* bfix2;               // 2D: the same at the last list build
    int4* bfix4;               // 3D; .w: its cell coordinates, x | y << 10 | z << 20
    uint32_t* bcxy;            // 2D: cell coordinates at the last list build, x | y << 16
    float2* boff;              // kReuseCell: offset from that cell's edges at the last list build
    uint32_t* slot;            // cell-order index at the last list build
    uint32_t* vl_far;          // non-zero: some particle is outside the grid (CellSplit::far); [1]: at the last rebuild
    uint32_t* vl_rebuild;      // non-zero: the next step rebuilds the grid and the lists
    uint32_t* vl_gone;         // the last build: bit 0 left out non-existent particles, bit 1 searched particles
    uint32_t* itype_changed;   // non-zero once a step changed a particle's type since the last upload
};

// A position in fixed point: 2^27 units a cell from the grid's origin, modulo 2^32
// (32 cells): the difference of two words is the separation of particles less
// than 16 cells apart. code carries the particle's kind in a float that is added to
// a squared distance: 0 fluid, -0 boundary, the smallest subnormal for other
// types; +inf absent (non-existent); NaN, low bits as before, for a particle
// outside the grid, which no list holds.
struct __align__(16) Pos {
    int x, y, z;
    float code;
#ifdef __CUDACC__
    __device__ __forceinline__ uint32_t bits() const { return __float_as_uint(code); }
    __device__ __forceinline__ bool absent() const { return bits() == 0x7F800000u; }
    __device__ __forceinline__ bool unlisted() const { return (bits() & 0x7FC00000u) == 0x7FC00000u; }
    __device__ __forceinline__ bool fluid() const { return (bits() & 0x80000001u) == 0u; }
    __device__ __forceinline__ bool boundary() const { return (int)bits() < 0; }
    static __device__ __forceinline__ float code_of(int32_t type, int32_t type_absent, bool far) {
        if (type == type_absent) return __uint_as_float(0x7F800000u);
        return __uint_as_float((type > 0 ? 0u : (type < 0 ? 0x80000000u : 1u)) | (far ? 0x7FC00000u : 0u));
    }
#endif
};

// Per-step cell-ordered copies and the grid.
struct Sorted {
    uint32_t *keys_in, *ids_in;       // key pass output (id order)
    uint32_t *keys_a, *ids_a, *keys_b, *ids_b;
    uint32_t* sort_scratch;
    uint32_t* scattered;              // counting sort: the ids grouped by cell, which the reorder puts in order (else null)
    uint32_t *key, *id;               // sorted result (points into a or b)
    uint32_t *cell_start, *cell_end;  // [max_cells]
    // FP64 gathers
    double *rx, *ry, *rz;
    double *vx, *vy, *vz;             // velocity the forces use (v_predict in the loop)
    double *vdx, *vdy, *vdz;          // velocity of density_con (v)
    double *rho;                      // density the forces use
    double *rhod;                     // density of density_con
    double* p;
    double* pr2;                      // p / (rho * rho) with the density the forces use (the density pass writes it)
    int32_t* itype;
    // FP32-mixed gathers
    float4* P4;    // cell-relative position (x, y, z) + itype bits
    float4* V4;    // velocity the forces use + density the forces use
    float4* VD4;   // v + (rho - rho0) for density_con
    float2* PR;    // pressure p and p / rho^2 (rho = the density the forces use)
    // mixed step with neighbour reuse: positions (in P4's buffer), with a row n of
    // an absent particle; and the positions / V4 (/ VD4 with continuity density) of
    // the next step, which the key pass writes at each particle's build slot (the
    // two buffers alternate)
    Pos* pos;
    Pos* posn;
    float4* V4n;
    float4* VD4n;
    // Neighbour masks written by the density pass for the force pass (the FP64
    // step, 2D and 3D; the 2D mixed step without reuse), SoA [NC + 1][n] with
    // NC = 3^dim stencil cells, of 32-bit words (64-bit in the 3D FP64 step):
    // word c < NC = bit b set if particle cell_start + b of stencil cell c is a
    // neighbour; word NC = stencil cells with more particles than a word has
    // bits (searched again by the force pass). Null where unused.
    uint32_t* nbmask;
    // stored-pair FP64 step (kernels_pairs64.cu; null elsewhere), cell order:
    double* pr;        // rows of 2 (3D: 4) doubles: position (3D: + density of the forces)
    double* pv;        // rows of 2 (4): velocity of the forces (3D: + p / rho^2)
    double* pq;        // 2D: rows of 2: density of the forces, p / rho^2
    double* pd;        // continuity density: rows of 2 (4): velocity v
    double* pe;        // delta-SPH: rows of 2: density rho, 1 / rho
    uint32_t* pnear;   // [3^dim][n], words as nbmask: the neighbours at up to one h, and some just beyond
    uint8_t* pbefore;  // [3^dim][n]: neighbours in the stencil cells before this one (at most 255)
    uint8_t* pown;     // [3^dim][n], summation density: the same of those with a larger sorted index (owned pairs)
    uint32_t* pcount;  // [n]: neighbours the masks hold
    uint32_t* pfirst;  // [3^dim][n]: first particle of the stencil cell
    double* pw;        // [cap][n], summation density: kernel value of neighbour number s
    double* pf;        // [cap][n] records of its acceleration: 2 doubles (2D summation density), or 4 with the rate
    double* ps;        // [cap][n], summation density: kernel gradient of owned pair number o
    uint8_t* prank;    // [cap][n]: its owner's number among the neighbours of the other particle
    // mixed step with neighbour reuse: up to kVerletCap2 (2D) / kVerletCap3 (3D)
    // candidates per particle as sorted indices, stored in slabs of four: entries
    // 4g..4g+3 of particle k are the uint4 at (uint4*)vlist + g * n + k (the lanes of
    // a warp read neighbouring uint4s), the last group padded with index n (an absent
    // particle); vcount[k] = candidates, or kListOver: the particle is searched
    // instead. This step's neighbours (the candidates within the cutoff, in list
    // order) in the same slab layout: nlist, ncount[k] of them; words past ncount are
    // stale. With split gathers (vl_split = 4) sub-list u of a particle takes the
    // groups u, u + 4, ... and ncount[k] holds four counts of 8 bits.
    uint32_t* vlist;
    uint32_t* vcount;
    uint32_t* nlist;
    uint32_t* ncount;
};

// Sources the reorder gathers for the force velocity / density.
struct GatherSrc {
    const double *vx, *vy, *vz;
    const double* rho;
    const double* p;  // pressure to copy (rrsph_forces on the given state); null in the loop
    int loop;         // 1: the loop's mixed step (float v_predict from the key pass; no double copies)
};

template <int DIM>
void launch_keys(const DevParams& P, const State& S, Sorted& G, StepScalars* scal, int predict, uint32_t* flags,
                 cudaStream_t st);
// for_whom: the gathers the cell-order copies are for.
enum : int { kReorderFp64 = 0, kReorderMixed = 1, kReorderPairs = 2, kReorderReuse = 3 };
template <int DIM>
void launch_reorder(const DevParams& P, const State& S, const Sorted& G, GatherSrc fsrc, int for_whom,
                    cudaStream_t st);
// The pair gathers take their block size (threads, <= kMaxGatherThreads, a
// multiple of 32) from the caller; the autotuner picks it.
template <int DIM>
void launch_density_fp64(const DevParams& P, const State& S, const Sorted& G, StepScalars* scal, uint32_t* flags,
                         cudaStream_t st, int threads);
// use_masks: the pairs are those the density pass on this grid recorded in
// G.nbmask (the same pairs in the same order as the search).
template <int DIM>
void launch_forces_fp64(const DevParams& P, const State& S, const Sorted& G, uint32_t terms, StepScalars* scal,
                        uint32_t* flags, int write_mu, cudaStream_t st, int threads, int use_masks = 0);
// The stored-pair FP64 step (kernels_pairs64.cu) on a grid reordered with kReorderPairs.
template <int DIM>
void launch_pair_masks(const DevParams& P, const State& S, const Sorted& G, StepScalars* scal, cudaStream_t st);
template <int DIM>
void launch_pair_terms(const DevParams& P, const Sorted& G, cudaStream_t st, int threads);
template <int DIM>
void launch_pair_density(const DevParams& P, const State& S, const Sorted& G, StepScalars* scal, uint32_t* flags,
                         cudaStream_t st);
template <int DIM>
void launch_pair_forces(const DevParams& P, const Sorted& G, cudaStream_t st, int threads);
template <int DIM>
void launch_pair_sum(const DevParams& P, const State& S, const Sorted& G, StepScalars* scal, uint32_t* flags,
                     cudaStream_t st);
template <int DIM>
void launch_density_mixed(const DevParams& P, const State& S, const Sorted& G, StepScalars* scal, uint32_t* flags,
                          cudaStream_t st, int threads);
template <int DIM>
void launch_forces_mixed(const DevParams& P, const State& S, const Sorted& G, uint32_t terms, StepScalars* scal,
                         uint32_t* flags, int write_mu, int use_masks, cudaStream_t st, int threads);
// whole_step; with next_keys also the next step's predict_half_step and key pass.
// pistons: a kernel of the step has evaluated the piston velocities (piston_block).
template <int DIM>
void launch_whole_step(const DevParams& P, const State& S, const Sorted& G, StepScalars* scal_cur,
                       StepScalars* scal_next, uint32_t* flags, int next_keys, cudaStream_t st, bool pistons = false);

// Neighbour reuse (the FP32-mixed step): the candidate lists
// are built with the cutoff widened by a skin and reused while no particle has
// moved more than half the skin since the build (kernels_reuse.cu).
void launch_verlet_decide(cudaGraphConditionalHandle h, const uint32_t* rebuild, cudaStream_t st);
void launch_verlet_reset(uint32_t* rebuild, uint32_t* gone, uint32_t* far, unsigned long long* builds,
                         cudaStream_t st);
// After an upload: the lists stay valid unless the last build left out a
// non-existent particle (which may exist now); moves are checked by the key pass.
void launch_verlet_upload_check(uint32_t* rebuild, const uint32_t* gone, cudaStream_t st);
template <int DIM>
void launch_verlet_build(const DevParams& P, const State& S, const Sorted& G, cudaStream_t st);
// Marks every cell-table entry empty (a kernel, so that it can sit in the
// rebuild body of a step graph's conditional node).
void launch_clear_cells(uint32_t* cell_start, uint32_t max_cells, cudaStream_t st);
// The last reuse step's neighbour list (nlist / ncount) as particle ids:
// counts[id], list[id * max_per + e]; more than max_per raises the overflow flag.
template <int DIM>
void launch_nlist_export(const DevParams& P, const Sorted& G, uint32_t* counts, uint32_t* list, uint32_t max_per,
                         uint32_t* flags, cudaStream_t st);
int verlet_split(int dim, uint32_t n);
template <int DIM>
void launch_density_verlet(const DevParams& P, const State& S, const Sorted& G, StepScalars* scal, uint32_t* flags,
                           cudaStream_t st, int threads);
// whole != 0: the whole step of each particle (launch_whole_step with next keys)
// runs in the force gather's thread; needs dt without the step's reduction and
// at most verlet_cap(dim) + 1 neighbours per particle (max_nb).
template <int DIM>
void launch_forces_verlet(const DevParams& P, const State& S, const Sorted& G, StepScalars* scal,
                          StepScalars* scal_next, uint32_t* flags, cudaStream_t st, int threads, int whole);

void launch_cells_start(const DevParams& P, const Sorted& G, uint32_t* out, cudaStream_t st);
template <int DIM>
void launch_neighbour_list(const DevParams& P, const Sorted& G, uint32_t* counts, uint32_t* list, uint32_t max_per,
                           uint32_t* flags, cudaStream_t st);
template <int DIM>
void launch_unpack(const DevParams& P, State S, const double* r, const double* v, uint32_t stride, cudaStream_t st);
template <int DIM>
void launch_pack(const DevParams& P, State S, double* r, double* v, uint32_t stride, cudaStream_t st);
// The time of the next step (and flags cleared, when non-null); after steps,
// the time and flags into a mapped host mailbox (device address `out`).
struct HostReport {
    double time;
    uint32_t flags;
    unsigned long long pairs_last;   // directed pairs of the last completed step (0: none since upload)
    unsigned long long pairs_total;  // summed over the steps since upload
};
void launch_set_time(StepScalars* scal, double time, uint32_t* flags, cudaStream_t st);
// rrsph_diagnostics: blocks partial sums of kDiagQuantities doubles into part
// (blocks * kDiagQuantities), then their fixed-order sum into out.
constexpr int kDiagQuantities = 10;
template <int DIM>
void launch_diagnostics(const DevParams& P, const State& S, double* part, int blocks, double* out, cudaStream_t st);
// scal: the next step's scalars; last: the completed step's (null: none since upload).
void launch_report(const StepScalars* scal, const StepScalars* last, const uint32_t* flags, HostReport* out,
                   cudaStream_t st);
// Upload / download through device-addressable host arrays (pinned memory):
// one kernel reading (writing) the caller's arrays over the host link. The
// upload also runs the first step's predict + key pass (launch_keys).
template <int DIM>
void launch_upload_direct(const DevParams& P, const State& S, const Sorted& G, const double* r, const double* v,
                          const double* rho, const double* p, const int32_t* itype, uint32_t stride,
                          StepScalars* scal, double dt, uint32_t* flags, cudaStream_t st);
// itype_if (optional): itype is written only if that device word is non-zero.
template <int DIM>
void launch_download_direct(const DevParams& P, const State& S, double* r, double* v, double* rho, double* p,
                            int32_t* itype, uint32_t stride, cudaStream_t st, const uint32_t* itype_if = nullptr);

// Stored values per particle of the FP64 pair sums: about 20 neighbours in 2D
// and 80 in 3D (120 to 160 beside the half-spaced walls); more are evaluated in place.
constexpr uint32_t kPairCap2 = 48;
constexpr uint32_t kPairCap3 = 160;
constexpr int kVerletCap2 = 64;         // candidate-list entries per particle, 2D
constexpr int kVerletCap3 = 256;        // and 3D
inline int verlet_cap(int dim) { return dim == 3 ? kVerletCap3 : kVerletCap2; }
// particles the reuse step takes
inline uint64_t verlet_max_particles(int dim) { return dim == 3 ? (1ull << 25) : (1ull << 27); }
// DevParams::reuse: fixed-point positions (kernels_reuse.cu), or cell-relative
// floats (kernels_reuse_cell.cu: 2D with split gathers), whose list entries hold a
// cell code above a 27-bit index.
enum : int { kReuseFixed = 1, kReuseCell = 2 };
constexpr uint32_t kCellEntryIndex = (1u << 27) - 1u;
constexpr uint32_t kListOver = 0xFFFFFFFFu;
constexpr int kGatherThreads = 128;     // default block size of the pair gathers
// ... of the 3D reuse gathers: bound by L1, which the warps of a block share
// (1.06M particles, us a step: 64 753, 128 717, 256 688)
constexpr int kReuseThreads3 = 256;
// ... of the stored-pair passes, whose warps meet nowhere: single warps, so that a
// block ends with its longest one (us a step at 32 / 64 / 128: 43k delta-SPH 93.1 /
// 96.9 / 98.7, 409k flume 476 / 479 / 480, 385k 3D 1988 / 1988 / 1993)
constexpr int kPairThreads = 32;
constexpr int kMaxGatherThreads = 256;

}  // namespace rrsph
