// gm_internal.cuh — definitions shared by the CUDA translation units of the
// GB300 backend: fixed-point force format, device status word, cell-grid
// description and the launchers each kernel file exports.
//
// Data layout in HBM (one system, N atoms):
//   * FP64 state in the caller's atom order: pos/vel/ref as x|y|z rows of N.
//   * int64 fixed-point force accumulators F (x|y|z rows, caller order),
//     value = F * 2^-40 kcal/mol/A.  Integer sums are associative, so
//     atomics from any thread order give bit-identical totals.
//   * Cell-sorted copies for the pair kernel: perm[s] = caller index of
//     sorted slot s; hi[s] = (x-o, y-o, z-o rounded to multiples of 2^-8 A,
//     Q_hi), lo[s] = (FP32 remainders of the same, Q_lo with the type in its
//     low 8 bits), Q = sqrt(k_C) q as a double-float; hi+lo carries each
//     coordinate to ~2^-33 A; FP64 mode keeps a sorted double4 copy.
//   * Full (symmetric) neighbour list in warp-interleaved columns: the 32
//     atoms of group g own a slab of 32*cap ints; entry e of lane l sits at
//     g*32*cap + e*32 + l, so one list row is a 128-byte coalesced load.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "geodesic_cuda.h"
#include "gm_df.h"
#include "gm_exact_math.h"

#define GM_FIX_SCALE 1099511627776.0        // 2^40
#define GM_FIX_INV (1.0 / 1099511627776.0)  // 2^-40
constexpr double GM_FORCE_TO_ACCEL = 20.455 * 20.455;  // kcal/mol/A/amu -> A/ps^2 (integrator.rs:9)
#define GM_FIX_SCALE_F 1099511627776.0f
#define GM_FIX_LIMIT 4194304.0              // 2^22: |contribution| must stay below

// Ceiling on distinct (sigma, epsilon) parameter pairs (the type sits in 8
// bits of a slot record; a single system's pair table of 16 B entries lives
// in shared memory while it fits in 48 KB, in L1 otherwise).
#define GM_MAX_TYPES 64
#define GM_WARP 32
#define GM_MAX_SPLIT 32      // largest number of work items per 32-atom group in the pair kernels
#define GM_SET_SPLIT 16      // largest split (parts of a group, each one or two work items) of a context
// The list build runs GM_NSEG warps per 32-atom group, one per z layer of the
// 5 x 5 x (span + 4) cell box the group's candidates come from (cells are at
// least half the list radius wide), or one per layer and y row.  Each warp
// stages the candidates its lanes accept, as masks over words of 32 candidates,
// in its own segment; the block then writes the segments' entries, one after
// the other, into each lane's list column.
#define GM_NSEG 5
// Threads per block of the bonded and 1-4 kernels.
#define GM_BONDED_THREADS 64
// List columns are ordered by build-time distance in GM_NBUCKET buckets.
#define GM_NBUCKET 4
#define GM_MAX_SLOTS ((1 << 27) - 1)  // padded atom slots of a context

// Device status bits (DevStatus::error).
enum : unsigned int {
    GM_DEV_NONFINITE_POS = 1u << 0,
    GM_DEV_NONFINITE_FORCE = 1u << 1,
    GM_DEV_FIX_OVERFLOW = 1u << 2,
    GM_DEV_LIST_OVERFLOW = 1u << 3,
    GM_DEV_SHAKE_FAIL = 1u << 4,
    GM_DEV_RATTLE_FAIL = 1u << 5,
    GM_DEV_EXTENT = 1u << 6,       // non-periodic extent too large for min-image
    GM_DEV_CELL_OVERFLOW = 1u << 7,
    GM_DEV_ITER_MISMATCH = 1u << 8,
    GM_DEV_BARRIER_TIMEOUT = 1u << 9,  // a grid barrier of the persistent step kernel gave up waiting
};

struct DevStatus {
    unsigned int error;
    unsigned int rebuild;          // 1 when the list must be rebuilt
    unsigned int blocks_done;      // last-block-done counter of the rebuild check
    unsigned int shake_T;          // iteration count of the last SHAKE call
    unsigned int rattle_T;
    unsigned int differs;          // uploaded positions differ from the resident ones
    unsigned long long n_rebuilds;
    unsigned long long step;       // current step of the resident loop
    unsigned long long fail_step;  // first step whose projection failed (init ~0)
    unsigned long long c_steps;    // resident steps with constraints
    unsigned long long shake_sum;  // sum of their SHAKE iteration counts
    unsigned long long rattle_sum; // sum of their RATTLE iteration counts
    unsigned int rec_n;            // warm-start samples recorded (in solves)
    unsigned int bad_pending;      // non-finite positions seen by the fused step kernel, moved to
                                   // error by its last block
    unsigned int max_count;        // largest list length the list build met (sizes a regrowth)
    unsigned int max_layer;        // largest staging (one z layer) length it met
    unsigned int tail_pending;     // unconstrained resident steps: the last step's closing half-kick
                                   // is still to do (the next step's first kernel or the finalizer)
    unsigned long long rebuild_base;  // n_rebuilds when the current call's status was reset
    unsigned int frame_n;          // trajectory frames recorded since they were last taken
    unsigned int frame_lost;       // frames due while the ring was full
    unsigned int stage_over;       // list groups whose staged words did not fit (built by the second kernel)
    unsigned long long c_loops;    // looping step launches run
};

struct GridInfo {
    double origin[3];   // coordinate origin of the float copies
    float lo[3];        // grid lower corner, origin-relative
    float inv_w[3];     // 1 / cell width
    float box[3], inv_box[3];
    int nc[3];
    int ncell;
    int periodic;
    int full[3];        // scan the whole dimension (periodic, fewer than 5 cells)
};

// ---------------------------------------------------------------- helpers

__device__ __forceinline__ long long gm_to_fix(double v) { return __double2ll_rn(v * GM_FIX_SCALE); }

// A float force contribution to fixed point; flags non-finite / overflow.
__device__ __forceinline__ long long gm_to_fix_checked(float v, unsigned int &bad) {
    if (!(fabsf(v) < (float)GM_FIX_LIMIT)) {
        bad |= isfinite(v) ? GM_DEV_FIX_OVERFLOW : GM_DEV_NONFINITE_FORCE;
        return 0;
    }
    return gm_f2fix(v);
}
__device__ __forceinline__ long long gm_to_fix_checked(double v, unsigned int &bad) {
    if (!isfinite(v)) bad |= GM_DEV_NONFINITE_FORCE;
    else if (fabs(v) >= GM_FIX_LIMIT) bad |= GM_DEV_FIX_OVERFLOW;
    return __double2ll_rn(v * GM_FIX_SCALE);
}

__device__ __forceinline__ void gm_atomic_fix_add(long long *p, long long v) {
    atomicAdd(reinterpret_cast<unsigned long long *>(p), static_cast<unsigned long long>(v));
}

// Per-system energies of a batch: int64 fixed point at 2^-32 kcal/mol, so the
// sum is independent of the order contributions arrive in.
constexpr double GM_EFIX_SCALE = 4294967296.0;

// Adds each lane's energy e to its system sy (sy < 0: nothing); one atomic
// per warp when the warp's lanes share a system.  All 32 lanes must call.
__device__ __forceinline__ void gm_add_sys_energy(long long *e_sys, int sy, double e) {
    const long long q = sy >= 0 ? __double2ll_rn(e * GM_EFIX_SCALE) : 0ll;
    const int s0 = __shfl_sync(0xffffffffu, sy, 0);
    if (__all_sync(0xffffffffu, sy == s0 || sy < 0) && s0 >= 0) {
        long long t = q;
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if ((threadIdx.x & 31) == 0) gm_atomic_fix_add(e_sys + s0, t);
    } else if (sy >= 0 && q != 0) {
        gm_atomic_fix_add(e_sys + sy, q);
    }
}

// Sum of x[0..n) over GM_SUM_BLOCKS blocks of 256 threads: this block's
// consecutive share, per-thread strided partial sums, then a tree over the
// block.  The last block to arrive (`last`, true for all its threads) adds the
// blocks' sums in a tree of its own.  The order is fixed, so every kernel that
// sums this way gets the same bits.  (One block alone took 13 us for the
// 33,000 partials of a 50,000-atom system: an FP64 addition holds a scheduler
// for 64 cycles.)
constexpr int GM_SUM_BLOCKS = 64;
__device__ __forceinline__ double gm_tree256(double v, double *s) {
    s[threadIdx.x] = v;
    __syncthreads();
    for (int k = 128; k > 0; k >>= 1) {
        if (threadIdx.x < k) s[threadIdx.x] += s[threadIdx.x + k];
        __syncthreads();
    }
    return s[0];
}
__device__ __forceinline__ double gm_share_sum256(const double *x, int n, double *s) {
    const int share = (n + GM_SUM_BLOCKS - 1) / GM_SUM_BLOCKS, b = blockIdx.x * share;
    const int e = b + share < n ? b + share : n;
    double acc = 0.0;
    for (int i = b + threadIdx.x; i < e; i += 256) acc += x[i];
    const double r = gm_tree256(acc, s);
    __syncthreads();
    return r;
}
// the blocks' sums, by one block (written before a __threadfence by the others)
__device__ __forceinline__ double gm_blocks_sum256(const double *part, double *s) {
    const double r = gm_tree256((int)threadIdx.x < GM_SUM_BLOCKS ? ((const volatile double *)part)[threadIdx.x] : 0.0, s);
    __syncthreads();
    return r;
}

// Fixed-order sum of all energy partials (pair items, bonded blocks, 1-4
// blocks) into the FP64 total: deterministic for a given launch shape.  Blocks
// 0..GM_SUM_BLOCKS-1 of the launch call it, 256 threads each, `s` 256 doubles.
__device__ __forceinline__ void gm_energy_block(const double *epart, int n, double *out, double *s) {
    __shared__ bool last;
    double *part = out + 1;
    unsigned *arrived = reinterpret_cast<unsigned *>(part + GM_SUM_BLOCKS);
    const double mine = gm_share_sum256(epart, n, s);
    if (threadIdx.x == 0) {
        part[blockIdx.x] = mine;
        __threadfence();
        last = atomicAdd(arrived, 1u) == GM_SUM_BLOCKS - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    const double e = gm_blocks_sum256(part, s);
    if (threadIdx.x == 0) {
        *out = e;
        *arrived = 0u;
    }
}

// Both float4 of a slot's (hi, lo) coordinate pair in one 256-bit load
// through the read-only path (the pair is 32-byte aligned).
__device__ __forceinline__ void gm_ld_coord(const float4 *p, float4 &h, float4 &l) {
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(h.x), "=f"(h.y), "=f"(h.z), "=f"(h.w), "=f"(l.x), "=f"(l.y), "=f"(l.z), "=f"(l.w)
        : "l"(p));
}
// The same where the launch itself writes the records (a launch of several
// steps reads what other blocks wrote before its last grid barrier).
__device__ __forceinline__ void gm_ld_coord_rw(const float4 *p, float4 &h, float4 &l) {
    asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(h.x), "=f"(h.y), "=f"(h.z), "=f"(h.w), "=f"(l.x), "=f"(l.y), "=f"(l.z), "=f"(l.w)
                 : "l"(p));
}

// A slot's atom type, kept in the low 8 bits of its Q_lo (the low part of a
// double-float charge; those bits are below 2^-39 of Q).
__device__ __forceinline__ int gm_slot_type(float qlo) { return __float_as_int(qlo) & 0xff; }

// Per atom: (Q_hi, Q_lo | type), Q = sqrt(k_C) q, built on the host.
// The slot record of an atom at FP64 offset (ox, oy, oz) from its system's
// grid origin: coordinates rounded to the 2^-8 A grid (differences of two
// such values, and their squares below 16 A, are exact in FP32) and the FP32
// remainders.
__device__ __forceinline__ void gm_pack_record(float4 *rec, double ox, double oy, double oz, float2 qw) {
    const float hx = rintf((float)ox * 256.f) * (1.f / 256.f);
    const float hy = rintf((float)oy * 256.f) * (1.f / 256.f);
    const float hz = rintf((float)oz * 256.f) * (1.f / 256.f);
    rec[0] = make_float4(hx, hy, hz, qw.x);
    rec[1] = make_float4((float)(ox - (double)hx), (float)(oy - (double)hy), (float)(oz - (double)hz), qw.y);
}
// One component of it: the grid value at rec[0], the remainder at rec[4].
__device__ __forceinline__ void gm_pack_component(float *rec, double o) {
    const float h = rintf((float)o * 256.f) * (1.f / 256.f);
    rec[0] = h;
    rec[4] = (float)(o - (double)h);
}

__device__ __forceinline__ unsigned gm_ld_acquire(const unsigned *p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// ~0.3 us per poll: 1.35 s before a block gives up (measured)
constexpr unsigned GM_BARRIER_POLLS = 1u << 22;

// Waits (one thread) until the barrier generation has left `g`; false, with the
// timeout recorded, when it did not within GM_BARRIER_POLLS polls.
__device__ __forceinline__ bool gm_wait_generation(const unsigned *gen, unsigned g, DevStatus *st) {
    for (unsigned it = 0; gm_ld_acquire(gen) == g; it++) {
        if (it >= GM_BARRIER_POLLS) {
            atomicOr(&st->error, (unsigned)GM_DEV_BARRIER_TIMEOUT);
            return false;
        }
        __nanosleep(64);
    }
    return true;
}

// Grid-wide barrier of a cooperative launch (every block is resident).  The
// generation is read before arriving, the last block to arrive resets the
// count and advances the generation.  Returns false (and records the
// timeout) when the generation did not advance within GM_BARRIER_POLLS polls.
// All threads of the block call.
__device__ __forceinline__ bool gm_grid_barrier(unsigned *arrive, unsigned *gen, DevStatus *st) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        int ok = 1;
        const unsigned g = gm_ld_acquire(gen);
        __threadfence();
        if (atomicAdd(arrive, 1u) == gridDim.x - 1) {
            atomicExch(arrive, 0u);
            __threadfence();
            atomicAdd(gen, 1u);
        } else {
            ok = gm_wait_generation(gen, g, st);
        }
        __threadfence();
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

// ------------------------------------------------------- launcher exports

struct ListArgs {
    int n;                   // atoms, all systems
    int n_slots;             // sorted slots: each system's atoms padded to a multiple of 32
    int n_sys;               // systems in the context
    int cap;                 // list entries per atom
    int cap_seg;             // staging entries per atom and z layer
    const double *pos;       // FP64 x|y|z rows of n atoms, caller order
    float4 *coord;           // per slot two float4 written by gm_pack_record
    double4 *pos64s;         // per slot FP64 copy (FP64 mode) or nullptr
    int *type_sorted;        // per slot types (FP64 mode)
    int *perm;               // slot -> atom (global index), -1 on padding slots
    int *slot_of;            // atom -> slot (or nullptr)
    int *cell_of;            // atom -> cell of its system
    int *cell_sorted;        // slot -> cell of its system
    int *cell_count, *cell_start, *cell_cursor;  // system s at sys_cell_off[s] (cell_start: ncell + 1 entries)
    int *tmp_atom;           // slot -> atom of the system, before the in-cell rank
    const int *type;         // caller order
    const float2 *qw;        // caller order: (Q_hi, Q_lo | type), see gm_pack_record
    const double *charge64;  // caller order (FP64 mode)
    const int *excl_start, *excl;   // caller-order CSR (both directions, sorted)
    int *list, *count, *gmax;
    int *count_in, *gmax_in;        // the same without the last distance bucket (the outer half of the skin)
    unsigned int *sys_far;          // nonzero: an atom of the system moved more than far_sq since its build (or nullptr)
    int *stage;              // [group][warp][word][4 rows][lane], cap_seg rows per layer
    double *ref;             // FP64 x|y|z copy at each system's build
    long long *force;        // zeroed with the pack
    GridInfo *grid;          // one per system
    DevStatus *status;
    double r_list, r_cut, r_switch, box[3];
    int periodic;
    double *bbox_scratch;    // [n_sys][bbox_blocks][9] (min, max, sum per dimension)
    int bbox_blocks, max_sys_atoms;
    // systems: atoms [sys_atom_off[s], +1), slots [sys_slot_off[s], +1) (32-aligned),
    // cells [sys_cell_off[s], +1) (the system's cell budget + 1)
    const int *sys_atom_off, *sys_slot_off, *sys_cell_off;
    const int *atom_sys;     // atom -> system
    const int *group_sys;    // 32-slot group -> system
    unsigned int *sys_flag;  // 1: rebuild the system's list at the next rebuild
};

// set (every system) or clear the rebuild flags; clearing also clears status->rebuild
void gm_launch_flags(const ListArgs &a, bool set, cudaStream_t s);
// `done` (or nullptr): nonzero for the systems to leave as they are.
void gm_launch_wrap(const ListArgs &a, double *pos, const unsigned int *done, cudaStream_t s);
void gm_launch_grid(const ListArgs &a, cudaStream_t s);
void gm_launch_bin(const ListArgs &a, cudaStream_t s);
// `all`: every system is marked.
void gm_launch_build(const ListArgs &a, bool all, cudaStream_t s);
// Whether that build splits a layer's y rows over warps.
bool gm_build_splits_rows(const ListArgs &a, bool all);
void gm_launch_pack(const ListArgs &a, bool fp64, cudaStream_t s);

// Constants of the mixed pair kernel; the low parts complete double-floats.
struct PairConst {
    float rc2, rsw2;          // cutoff^2, switch radius^2 (FP32 tests)
    float rsw, rsw_lo;        // switch radius
    float inv_w, inv_w_lo;    // 1 / (cutoff - switch radius)
    float mds, mds_lo;        // -30 / (cutoff - switch radius): dS/dr = mds u^2 (1 - u)^2
    float box[3], box_lo[3], inv_box[3];
    float img2;               // raw squared distances up to it need no image: (0.49 box)^2
};

struct ForceArgs {
    int n, n_groups, cap;
    int n_slots;             // n_groups * 32 (each system padded to whole groups)
    const int *group_sys, *atom_sys;
    long long *e_sys;        // per-system potential energy, fixed point 2^-32 kcal/mol (batches), or nullptr
    int split;               // work items per 32-atom group in the pair kernels
    int quad;                // the persistent kernel gives a pair item a block (small systems)
    int term_chunk;          // bonded terms (or 1-4 pairs) per work item of the persistent kernel
    int pair_warps;          // warps per block of the FP32 pair kernel (2, 4, 8)
    int pair_grid;           // blocks of the FP32 pair kernel (0: one work item per warp; fewer: persistent)
    const float4 *coord;     // per slot (hi, lo) pairs: one 32-byte sector per gathered atom
    const double4 *pos64s;
    const int *type_sorted;  // FP64 mode
    const int *perm;
    const int *list, *count, *gmax;
    // While no atom of a system has moved more than a quarter of the skin (less
    // 1e-3 A) since its build, pairs of the last distance bucket (beyond half
    // the skin) cannot be inside the cutoff, and the columns end before them.
    // sys_far[system] != 0 (or nullptr: unknown) takes the whole columns.  Mixed
    // kernels only: an FP64 entry past the cutoff costs an FP32 test, less than
    // the look at the flag (5,000 atoms: 2 % slower with it).
    const int *count_in, *gmax_in;
    const unsigned int *sys_far;
    int ntypes;
    const float4 *tab32;     // (sigma_ij^2, 24 epsilon_ij) per type pair, each a double-float (hi, lo)
    const double2 *tab64;    // (sigma_ij^2, 24 epsilon_ij), or zeros where epsilon_ij is 0
    PairConst pc;            // the mixed pair kernel's constants
    double rc2_64, rsw_64, inv_wsw_64;
    float rc2_pre;           // FP64 kernel's FP32 pre-test: beyond it a pair is outside the cutoff for certain
    int coulomb;
    float box[3], inv_box[3];
    double box64[3];
    int periodic;
    int bonded_mi;  // periodic && bonded_min_image: bonded and 1-4 differences at the nearest image
    long long *force;
    double *epart;           // per pair-kernel warp (n_groups * split), then bonded, then 1-4
    DevStatus *status;
    const double *pos;       // caller order FP64 (bonded)
    // bonded, caller order
    int n_bonds, n_angles, n_diheds;
    const int *bond_i, *bond_j; const double *bond_k, *bond_r0;
    const int *angle_i, *angle_j, *angle_k; const double *angle_kth, *angle_th0;
    const int *dihed_i, *dihed_j, *dihed_k, *dihed_l; const double *dihed_kphi; const int *dihed_n;
    const double *dihed_delta;
    const double2 *dihed_cs;  // (cos delta, sin delta) per dihedral
    double *epart_bonded;    // per block
    int bonded_blocks;
    // scaled 1-4 pairs
    int n14; const int *p14_i, *p14_j; double scale14_lj, scale14_coul;
    const double *sigma, *epsilon, *charge64;
    const double4 *p14par;   // per 1-4 pair: (sigma_ij, 4 eps_ij s_lj, 24 eps_ij s_lj, k_C q_i q_j s_coul)
    double *epart14; int blocks14;
    double *energy;          // total, then GM_SUM_BLOCKS block sums and the arrival count of their sum
    int n_epart_total;       // n_groups * split + bonded_blocks + blocks14 entries
};

void gm_launch_pair(const ForceArgs &a, bool fp64, cudaStream_t s);
void gm_launch_bonded(const ForceArgs &a, bool fp64, cudaStream_t s);
void gm_launch_pair14(const ForceArgs &a, bool fp64, cudaStream_t s);
// the bonded terms and the 1-4 pairs in one launch
void gm_launch_bonded_pair14(const ForceArgs &a, bool fp64, cudaStream_t s);
void gm_launch_energy(const ForceArgs &a, cudaStream_t s);
int gm_bonded_blocks(int n_bonds, int n_angles, int n_diheds);

struct ClusterArgs {
    int n_clusters;
    int n_star_end;                       // clusters [0, n_star_end): 1-8 constraints sharing one centre atom
    int n_warp_end;                       // [n_star_end, n_warp_end): other clusters, 2-32 constraints, <= 32 atoms
    // the stars' lanes, 32 per warp, each star on 1, 2, 4 or 8 aligned lanes
    // of a warp of that width: (centre, other atom, constraint or -1, cluster or -1)
    int n_lane_warps;
    const int4 *lanes;
    const int *lane_width;                // per warp
    const int *cl_cstart, *cl_cons;       // cluster -> constraints (ascending)
    const int *cl_astart, *cl_atoms;      // cluster -> atoms
    const int *cl_acstart, *cl_acons;     // cluster-atom slot -> signed constraint refs (ascending)
    const int *constr_i, *constr_j;
    const double *constr_dsq;
    const double *inv_mass;               // 1.0 / mass (caller order)
    double *lam;                          // per constraint scratch
    double *lam_sum;                      // per constraint accumulated multiplier (nullptr: not kept)
    const double *lam0;                   // per constraint warm-start multiplier (nullptr: cold start)
    double *rvec;                         // per constraint reference vector (3 x C)
    int *cl_iters;                        // per cluster iteration count
    double *cl_worst;                     // per cluster last max |lambda|
    int *cl_worst_idx;                    // per cluster constraint of that max
    int n_constr;
    unsigned int max_iter;
    double tol;
    DevStatus *status;
    int mi;                               // constraint differences at the nearest image of box64
    double box64[3];
};

void gm_launch_half_kick(int n, double *vel, const long long *force, const double *inv_mass, double dt_half,
                         const DevStatus *st, cudaStream_t s);
void gm_launch_half_kick_f64(int n, double *vel, const double *force, const double *inv_mass, double dt_half,
                             cudaStream_t s);
void gm_launch_drift(int n, double *pos, double *vel, double *dref, double dt, bool resync, const DevStatus *st,
                     cudaStream_t s);
void gm_launch_resync(int n, const double *pos, double *vel, const double *dref, double dt, const DevStatus *st,
                      cudaStream_t s);
void gm_launch_check(int n, const double *pos, const double *ref, double thr_sq, double far_sq, DevStatus *st,
                     unsigned long long cond_handle, int blocks, const int *atom_sys, unsigned int *sys_flag,
                     unsigned int *sys_far, cudaStream_t s);
void gm_launch_shake(const ClusterArgs &c, int n_atoms, const double *dref, double *pos, cudaStream_t s);
// the same solve in two halves, so the warm start can run in between:
// prepare (reset T, reference vectors, multiplier sums) and the iterations
// (warm-start displacement when c.lam0 is set, then both phases)
void gm_launch_shake_prepare(const ClusterArgs &c, int n_atoms, const double *dref, cudaStream_t s);
int gm_launch_shake_solve(const ClusterArgs &c, int n_atoms, double *pos, cudaStream_t s);
// `reset`: clear rattle_T first (a status reset has cleared it already).
void gm_launch_rattle(const ClusterArgs &c, int n_atoms, const double *pos, double *vel, bool reset, cudaStream_t s);
void gm_launch_step(DevStatus *st, cudaStream_t s);
// Unconstrained step: half-kicks (the previous step's closing one and this
// step's opening one) + drift (with the velocity resync) + rebuild check +
// coordinate pack in one launch.  Each atom gets the same operations in the
// same order as the separate kernels.
// The pack kernel's per-atom work (FP32 (hi, lo) copies relative to the
// system's grid origin, FP64 copies in FP64 mode, forces cleared), done by the
// fused step kernel for the force evaluation that follows it.
struct PackArgs {
    float4 *coord;
    double4 *pos64s;
    int *type_sorted;
    const int *slot_of;
    const GridInfo *grid;
    const int *type;
    const float2 *qw;
    const double *charge64;
    int fp64;
};
// The persistent step kernel (gm_step.cu): one cooperative launch per
// unconstrained mixed-precision step.  Its force phase hands out work items
// (pair items and 32-term bonded / 1-4 chunks) from `ticket`; one grid
// barrier separates it from the kick / drift / rebuild check / pack phase.
struct StepSync {
    unsigned int arrive;  // blocks arrived at the grid barrier
    unsigned int gen;     // barrier generation
    unsigned int ticket;  // next work item of the force phase
    unsigned int fresh;   // nonzero: the forces at the current positions are summed already (skip the phase)
    unsigned int more;    // the launch goes on with another step
    unsigned int pad;
    long long todo;       // looping launches: steps left in the call
};
// Steps a looping launch runs at most before its graph's WHILE node asks again.
constexpr int GM_LOOP_STEPS = 64;
struct StepArgs {
    int n;
    double *pos, *vel, *dref;
    const double *inv_mass, *ref;
    double dt_half, dt, inv_dt, thr_sq, far_sq;
    unsigned long long cond;   // graph conditional handle of the rebuild, or 0
    unsigned long long loop;   // handle of the WHILE node round a launch of up to GM_LOOP_STEPS steps; 0: one step
    const int *atom_sys;
    unsigned int *sys_flag, *sys_far;
    StepSync *sync;
};
// The constrained step's two cooperative kernels (star clusters only):
//   shake: half-kick, drift, SHAKE, velocity resync, rebuild check, pack;
//   rattle: half-kick, RATTLE, the step count.
// Both phases of a solve run in one launch with a grid barrier between them.
struct SolveSync {
    unsigned int arrive, gen;  // grid barrier
    unsigned int T;            // largest iteration count of phase 1
    unsigned int fail;         // a cluster of phase 1 did not converge
    long long todo;            // RATTLE's: steps left in the call
};
struct SolveStepArgs {
    int n, n_free;
    const int *free_atoms;     // atoms of no constraint
    double *pos, *vel, *dref;
    long long *force;
    const double *ref;
    double dt_half, dt, inv_dt, thr_sq, far_sq;
    unsigned long long loop;   // handle of the WHILE node round the step, or 0
    unsigned long long cond;
    const int *atom_sys;
    unsigned int *sys_flag, *sys_far;
    SolveSync *sync;
};
// Threads per block and blocks (all co-resident) of both kernels; blocks 0
// when the system's clusters do not fit.
void gm_solve_step_grid(const ClusterArgs &c, int n_free, int *threads, int *blocks, bool *quads);
// Clears the two solves' words; `todo`: the steps of the call.
void gm_launch_solve_begin(SolveSync *two, long long todo, cudaStream_t s);
void gm_launch_shake_step(const ClusterArgs &c, const SolveStepArgs &sa, const PackArgs &pk, int threads, int blocks,
                          bool quads, cudaStream_t s);
void gm_launch_rattle_step(const ClusterArgs &c, const SolveStepArgs &sa, int threads, int blocks, bool quads,
                           cudaStream_t s);
// Blocks of the cooperative grid (all co-resident, no more than the work
// items and atoms fill); 0 when the form does not apply.
int gm_step_persistent_blocks(const ForceArgs &fa);
void gm_launch_step_persistent(const ForceArgs &fa, const StepArgs &sa, const PackArgs &pk, int blocks,
                               cudaStream_t s);
// Whether the step kernel of these arguments can run several steps a launch.
bool gm_step_loops(const ForceArgs &a);
// Clears the step's words; `fresh`: the forces are summed already; `todo`: the
// steps of the call.
void gm_launch_step_begin(StepSync *sync, bool fresh, long long todo, cudaStream_t s);
// The persistent kernel's force phase alone, with energies (the force
// kernels' partials, the same bits), as a plain launch: pair items and bonded
// / 1-4 blocks from one queue.  The queue words must be zero.
void gm_launch_forces_persistent(const ForceArgs &fa, StepSync *sync, int blocks, cudaStream_t s);
void gm_launch_kick_drift_check(int n, double *pos, double *vel, double *dref, long long *force,
                                const double *inv_mass, double dt_half, double dt, const double *ref, double thr_sq,
                                double far_sq, DevStatus *st, unsigned long long cond, const int *atom_sys,
                                unsigned int *sys_flag, unsigned int *sys_far, const PackArgs &pk, cudaStream_t s);
// Trajectory frames recorded on the device during resident steps.
struct FrameArgs {
    int interval;                // a frame when the completed step count is a multiple (0: none)
    int cap;                     // frames the ring holds
    float *xyz;                  // [cap][3][n] positions as float32
    unsigned long long *step;    // [cap] step of each frame
    double *energy;              // [cap][2] potential and kinetic energy (kcal/mol)
    double *partial;             // [2][GM_FRAME_BLOCKS] kinetic and potential partial sums
    const double *epart;         // energy partials of the last force evaluation
    int n_epart;
};
constexpr int GM_FRAME_BLOCKS = GM_SUM_BLOCKS;  // the kinetic reduction's grid (as gm_kinetic_energy's)
// Records a frame when the step just completed is due: positions as float32,
// the kinetic energy of the step's final velocities (its closing half-kick
// applied when still pending, in the finalizer's arithmetic; the reduction of
// gm_kinetic_energy) and the potential energy (the energy kernel's sum).
void gm_launch_frame(int n, const double *pos, const double *vel, const long long *force, const double *inv_mass,
                     const double *mass, double dt_half, DevStatus *st, const FrameArgs &f, cudaStream_t s);
// The closing half-kick and step count of the last unconstrained resident
// step, when one is pending (a no-op otherwise).
// With `epart` the launch sums the n_epart energy partials into `energy` too.
void gm_launch_kick_tail(int n, double *vel, const long long *force, const double *inv_mass, double dt_half,
                         DevStatus *st, const double *epart, int n_epart, double *energy, cudaStream_t s);
void gm_launch_kinetic(int n, const double *vel, const double *mass, double *partials, int blocks, double *out,
                       cudaStream_t s);
void gm_launch_forces_out(int n, const long long *force, double *out, cudaStream_t s);
void gm_launch_differs(int n, const double *a, const double *b, unsigned int *flag, cudaStream_t s);
// The per-call status reset on the device: counters kept, per-call fields
// cleared, the step set when set_step, n_rebuilds noted as the call's base
// unless keep_base.
void gm_launch_status_reset(DevStatus *st, int set_step, unsigned long long step, int keep_base, cudaStream_t s);
int gm_check_blocks(int n);

// ---- constraint warm start (gm_mlp.cu) -----------------------------------
// A 12-64-64-1 SiLU network over per-constraint features predicts the
// constraint's total SHAKE multiplier, as a correction to the first Jacobi
// step (t = Lambda * 2 (1/m_i + 1/m_j) = t1 + network).  FP32 master parameters, laid out as
// W1[12][64], b1[64], W2[64][64], b2[64], w3[64], b3; the matmul weights and
// the activations are rounded to BF16, sums are FP32.  norm holds the
// feature means[12], feature scales[12], target mean, target scale.
constexpr int GM_WS_IN = 12, GM_WS_H = 64;
constexpr int GM_WS_OFF_W1 = 0, GM_WS_OFF_B1 = 768, GM_WS_OFF_W2 = 832, GM_WS_OFF_B2 = 4928, GM_WS_OFF_W3 = 4992,
              GM_WS_OFF_B3 = 5056, GM_WS_NPAR = 5057, GM_WS_NNORM = 26;
constexpr int GM_WS_TILE = 128;  // samples per block of the training kernel

// Features of constraint k = (i, j), d0^2 = dsq, r = ref_i - ref_j, d =
// trial_i - trial_j, w = 1/m_i + 1/m_j:
//  0 (d.d - d0^2) / d0^2   1 d.r / d0^2   2 d0   3 1/m_i   4 1/m_j
//  5, 6 constraints on i, on j   7 t1 = (d.d - d0^2) / d.r (the first Jacobi
//  step times 2 w)   8 c1 = sum over the other constraints l on a shared
//  atom a of (1/m_a) / w_k cos(r_k, r_l) s_k s_l t1_l w_k / w_l (the first
//  order coupling; s = +1 where a is the constraint's i, -1 where it is j)
//  9 sum of the squared coupling coefficients   10 max |cos|   11 sum of t1_l
//  (8-11 in FP32)
struct WsFeatureArgs {
    int n_constr, n_atoms;
    const int *constr_i, *constr_j;
    const double *constr_dsq, *inv_mass;
    const int *atom_cstart, *atom_cref;  // per-atom constraints (CSR; ref k: atom is i, -k-1: atom is j)
    const double *pos, *dref;    // trial and reference positions
    float *feat;                 // [n_constr][12] raw features
    double *scale;               // 2 (1/m_i + 1/m_j) per constraint
    double *t1;                  // first Jacobi step of a cold solve, times scale
    float4 *unit;                // (reference bond direction, t1) per constraint (FP32), for the coupling pass
    const float *w;              // 1/m_i + 1/m_j per constraint, FP32 (each mass rounded first)
};
// Two launches per solve: every constraint's raw features, t1 and scale, and
// with infer the network on the tensor cores (fused with the coupling pass)
// and the predicted multipliers lam0[k] = (t1[k] + y_k * t_scale + t_mean) /
// scale[k].  `packed`: the parameters and standardisation as gm_launch_ws_pack
// left them.
void gm_launch_ws_predict(const WsFeatureArgs &a, const void *packed, double *lam0, bool infer, cudaStream_t s);
// The inference's parameter block (gm_ws_packed_bytes bytes), written from
// the parameters and the input standardisation; run after every change of
// either.
size_t gm_ws_packed_bytes();
void gm_launch_ws_pack(const float *params, const float *norm, void *packed, cudaStream_t s);
// The network's output y for m standardised inputs x[m][12] (same kernels).
void gm_launch_ws_forward(int m, const float *x, const float *params, float *y, cudaStream_t s);
// records raw features and targets lam_sum * scale - t1 into slot rec_n when
// step % stride == 0 (resident steps), then advances rec_n
void gm_launch_ws_record(int n_constr, const float *feat, const double *lam_sum, const double *scale, const double *t1,
                         float *rec_feat, float *rec_t, int stride, int cap_slots, DevStatus *st, cudaStream_t s);
// feature/target statistics over n samples into norm (device, deterministic)
void gm_launch_ws_stats(long long n, const float *feat, const float *t, double *partial, int blocks, float *norm,
                        cudaStream_t s);
// one forward/backward pass over a batch of blocks x 128 samples; sample b*128+s
// is idx ? idx[...] : hash(seed, iter, .) % n.  Writes per-block gradients
// and loss into partial[blocks][NPAR + 1]; rows past n_valid count nothing.
void gm_launch_ws_grad(long long n, const float *feat, const float *t, const float *norm, bool standardized,
                       const float *params, int blocks, unsigned long long seed, long long iter, long long n_valid,
                       float *partial, cudaStream_t s);
// fixed-order sum of the block gradients; Adam step when m != nullptr,
// otherwise the summed gradient (and loss) go to grad_out
void gm_launch_ws_update(int blocks, const float *partial, float *params, float *m, float *v, float lr, float b1,
                         float b2, float eps, int t, float *grad_out, cudaStream_t s);
