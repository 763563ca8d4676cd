// gm_integrate_exact.cu — FP64 integrator and constraint kernels.
//
// Built with --fmad=false: every expression below rounds after each
// operation in the order written, like the reference's Rust (which never
// contracts a*b+c).  Given the same forces, half-kick, drift and the
// SHAKE/RATTLE projections therefore return the reference's exact bits.
//
// Constraint solver (constraint.rs:62-152, :170-259).  The reference sweeps
// every constraint per Jacobi iteration and stops when max|lambda| < tol
// over all of them.  Constraints only couple through shared atoms, so the
// work splits into independent clusters (connected components of the
// constraint graph, found once on the host): a star has a lane per constraint
// (or four), another cluster a warp, a large one a thread.
// Phase 1 iterates each cluster until its own max|lambda| < tol and records
// its count t_c; the global count is T = max t_c (the first iteration where
// every cluster is below tol, given that a converged cluster stays below
// tol).  Phase 2 advances every cluster to exactly T iterations and checks
// that assumption at iteration T (flagging GM_DEV_ITER_MISMATCH otherwise).
// Within a cluster, per-atom deltas are summed over the atom's constraints in
// ascending constraint index, starting from 0.0, as the reference's
// delta_x/y/z arrays are; positions after T iterations are bit-identical.
#include "gm_internal.cuh"

namespace {

constexpr double kForceToAccel = GM_FORCE_TO_ACCEL;  // integrator.rs:9

__global__ void half_kick_kernel(int n, double *vel, const long long *force, const double *inv_mass, double dt_half,
                                 const DevStatus *st) {
    // integrator.rs:14-21: v += dt_half * F * inv_m * 20.455^2
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || st->error) return;
    const double inv_m = inv_mass[i];
    for (int d = 0; d < 3; d++) {
        const double f = (double)force[d * n + i] * GM_FIX_INV;
        vel[d * n + i] += dt_half * f * inv_m * kForceToAccel;
    }
}

__global__ void half_kick_f64_kernel(int n, double *vel, const double *force, const double *inv_mass, double dt_half) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double inv_m = inv_mass[i];
    for (int d = 0; d < 3; d++) vel[d * n + i] += dt_half * force[d * n + i] * inv_m * kForceToAccel;
}

__global__ void drift_kernel(int n, double *pos, double *vel, double *dref, double dt, int resync,
                             const DevStatus *st) {
    // integrator.rs:32-48 (and :64-68 when no constraint can move the atom)
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || st->error) return;
    for (int d = 0; d < 3; d++) {
        const double p = pos[d * n + i];
        const double v = vel[d * n + i];
        dref[d * n + i] = p;
        const double np = p + dt * v;
        pos[d * n + i] = np;
        if (resync) vel[d * n + i] = (np - p) / dt;
    }
}

__global__ void resync_kernel(int n, const double *pos, double *vel, const double *dref, double dt, double inv_dt,
                              const DevStatus *st) {
    // integrator.rs:64-68 (skipped after a failed projection, like the `?` at integrator.rs:256)
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || st->error) return;
    for (int d = 0; d < 3; d++) vel[d * n + i] = gm_div_by_dt(pos[d * n + i] - dref[d * n + i], dt, inv_dt);
}

__global__ void check_kernel(int n, const double *pos, const double *ref, double thr_sq, double far_sq, DevStatus *st,
                             unsigned long long cond, const int *atom_sys, unsigned int *sys_flag,
                             unsigned int *sys_far) {
    // neighbor.rs:60-72 plus the run loop's finite-position guard (lib.rs:94-107);
    // the atom's system is marked for the rebuild
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    int need = 0, bad = 0;
    if (i < n) {
        const double x = pos[i], y = pos[n + i], z = pos[2 * n + i];
        bad = !(isfinite(x) && isfinite(y) && isfinite(z));
        const double dx = x - ref[i], dy = y - ref[n + i], dz = z - ref[2 * n + i];
        const double d2 = dx * dx + dy * dy + dz * dz;
        need = d2 > thr_sq;
        if (need) sys_flag[atom_sys[i]] = 1u;
        if (gm_moved_far(d2, far_sq)) sys_far[atom_sys[i]] = 1u;
    }
    need = __syncthreads_or(need);
    bad = __syncthreads_or(bad);
    if (threadIdx.x == 0) {
        if (need) atomicOr(&st->rebuild, 1u);
        if (bad) atomicOr(&st->error, (unsigned)GM_DEV_NONFINITE_POS);
        __threadfence();
        const unsigned done = atomicAdd(&st->blocks_done, 1u);
        if (done == gridDim.x - 1) {
            // last block: every block's flag is visible now
            __threadfence();
            const unsigned r = atomicOr(&st->rebuild, 0u);
            st->blocks_done = 0;
            // never rebuild from a failed state (NaN positions would pile into one cell)
            const unsigned e = atomicOr(&st->error, 0u);
            if (cond) cudaGraphSetConditional((cudaGraphConditionalHandle)cond, (r && !e) ? 1u : 0u);
        }
    }
}

// The position difference a - b along axis d of a constraint: raw (the
// reference), or at the nearest periodic image when c.mi (bonded_min_image).
// Exact arithmetic (this file builds without FMA contraction), so the raw
// difference is the same bits as before the option existed and the image
// form those of the restated min_image.
__device__ __forceinline__ double cdiff(const ClusterArgs &c, double a, double b, int d) {
    const double v = a - b;
    return c.mi ? gm_min_image(v, c.box64[d]) : v;
}

// One Jacobi iteration over a cluster.  Returns max|lambda| and its
// constraint (first in ascending order, as the reference's strict '>').
__device__ void shake_iteration(const ClusterArgs &c, int cl, const double *rvec, double *pos, int n_atoms,
                                double &max_out, int &worst_out) {
    const int c0 = c.cl_cstart[cl], c1 = c.cl_cstart[cl + 1];
    double max_lambda = 0.0;
    int worst = c0 < c1 ? c.cl_cons[c0] : 0;
    const int nc = c.n_constr;
    for (int q = c0; q < c1; q++) {
        const int k = c.cl_cons[q];
        const int i = c.constr_i[k], j = c.constr_j[k];
        const double dx = cdiff(c, pos[i], pos[j], 0);
        const double dy = cdiff(c, pos[n_atoms + i], pos[n_atoms + j], 1);
        const double dz = cdiff(c, pos[2 * n_atoms + i], pos[2 * n_atoms + j], 2);
        const double diff = dx * dx + dy * dy + dz * dz - c.constr_dsq[k];
        const double rx = rvec[k], ry = rvec[nc + k], rz = rvec[2 * nc + k];
        const double inv_mi = c.inv_mass[i], inv_mj = c.inv_mass[j];
        const double dot_new_old = dx * rx + dy * ry + dz * rz;
        const double denom = 2.0 * (inv_mi + inv_mj) * dot_new_old;
        const double lambda = denom == 0.0 ? 0.0 : diff / denom;
        c.lam[k] = lambda;
        if (c.lam_sum) c.lam_sum[k] += lambda;  // the multiplier total, lam0 + sum of iterations
        const double la = fabs(lambda);
        if (la > max_lambda) { max_lambda = la; worst = k; }
    }
    const int a0 = c.cl_astart[cl], a1 = c.cl_astart[cl + 1];
    for (int q = a0; q < a1; q++) {
        const int a = c.cl_atoms[q];
        const double inv_m = c.inv_mass[a];
        double ddx = 0.0, ddy = 0.0, ddz = 0.0;
        for (int r = c.cl_acstart[q]; r < c.cl_acstart[q + 1]; r++) {
            const int ref = c.cl_acons[r];
            const int k = ref >= 0 ? ref : -ref - 1;   // negative: atom is constraint's i
            const double w = c.lam[k] * inv_m;
            const double tx = w * rvec[k], ty = w * rvec[nc + k], tz = w * rvec[2 * nc + k];
            if (ref < 0) { ddx -= tx; ddy -= ty; ddz -= tz; }
            else { ddx += tx; ddy += ty; ddz += tz; }
        }
        pos[a] += ddx;
        pos[n_atoms + a] += ddy;
        pos[2 * n_atoms + a] += ddz;
    }
    max_out = max_lambda;
    worst_out = worst;
}

__device__ void rattle_iteration(const ClusterArgs &c, int cl, const double *pos, double *vel, int n_atoms,
                                 double &max_out, int &worst_out) {
    const int c0 = c.cl_cstart[cl], c1 = c.cl_cstart[cl + 1];
    double max_mu = 0.0;
    int worst = c0 < c1 ? c.cl_cons[c0] : 0;
    const int nc = c.n_constr;
    for (int q = c0; q < c1; q++) {
        const int k = c.cl_cons[q];
        const int i = c.constr_i[k], j = c.constr_j[k];
        const double rx = cdiff(c, pos[i], pos[j], 0);
        const double ry = cdiff(c, pos[n_atoms + i], pos[n_atoms + j], 1);
        const double rz = cdiff(c, pos[2 * n_atoms + i], pos[2 * n_atoms + j], 2);
        const double rsq = rx * rx + ry * ry + rz * rz;
        const double dvx = vel[i] - vel[j];
        const double dvy = vel[n_atoms + i] - vel[n_atoms + j];
        const double dvz = vel[2 * n_atoms + i] - vel[2 * n_atoms + j];
        const double rel_vel = dvx * rx + dvy * ry + dvz * rz;
        const double inv_mi = c.inv_mass[i], inv_mj = c.inv_mass[j];
        const double denom = (inv_mi + inv_mj) * rsq;
        const double mu = denom == 0.0 ? 0.0 : rel_vel / denom;
        c.lam[k] = mu;
        c.rvec[k] = rx;
        c.rvec[nc + k] = ry;
        c.rvec[2 * nc + k] = rz;
        const double ma = fabs(mu);
        if (ma > max_mu) { max_mu = ma; worst = k; }
    }
    const int a0 = c.cl_astart[cl], a1 = c.cl_astart[cl + 1];
    for (int q = a0; q < a1; q++) {
        const int a = c.cl_atoms[q];
        const double inv_m = c.inv_mass[a];
        double ddx = 0.0, ddy = 0.0, ddz = 0.0;
        for (int r = c.cl_acstart[q]; r < c.cl_acstart[q + 1]; r++) {
            const int ref = c.cl_acons[r];
            const int k = ref >= 0 ? ref : -ref - 1;
            const double w = c.lam[k] * inv_m;
            const double tx = w * c.rvec[k], ty = w * c.rvec[nc + k], tz = w * c.rvec[2 * nc + k];
            if (ref < 0) { ddx -= tx; ddy -= ty; ddz -= tz; }
            else { ddx += tx; ddy += ty; ddz += tz; }
        }
        vel[a] += ddx;
        vel[n_atoms + a] += ddy;
        vel[2 * n_atoms + a] += ddz;
    }
    max_out = max_mu;
    worst_out = worst;
}

// Reference vectors r_ref = ref_i - ref_j (constraint.rs:106-108), fixed for the call.
__global__ void shake_prepare(ClusterArgs c, const double *dref, int n_atoms) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= c.n_constr) return;
    const int i = c.constr_i[k], j = c.constr_j[k];
    c.rvec[k] = cdiff(c, dref[i], dref[j], 0);
    c.rvec[c.n_constr + k] = cdiff(c, dref[n_atoms + i], dref[n_atoms + j], 1);
    c.rvec[2 * c.n_constr + k] = cdiff(c, dref[2 * n_atoms + i], dref[2 * n_atoms + j], 2);
    if (c.lam_sum) c.lam_sum[k] = 0.0;
}

// Star clusters: 1-8 constraints that all share one centre atom (a heavy atom
// and its H atoms; a single constraint is a star of one).  One constraint per
// lane: a star has a group of 1, 2, 4 or 8 lanes, each with its own H atom and
// multiplier in registers and a copy of the centre, which all of them update
// alike from the group's shuffled terms.  The operations are those of the
// general sweep in the same order: each constraint's multiplier, then each
// atom's sum over its constraints (the centre's in ascending constraint order,
// from 0.0).  Differences are taken centre minus H whichever atom is the
// constraint's i: both signs flip in every product, so the values are the
// same bits.
// An iteration is one serial chain of FP64 operations whatever the star's
// size, 64 cycles of its scheduler each, so what need not be FP64 is not: the
// convergence and zero tests compare bits, RATTLE's division by its constant
// denominator is three operations from the reciprocal, and the centre's sum
// starts from the first term.  With a thread per star it was that for every
// constraint of the star, and the one warp holding the four-H stars of a
// 20,011-atom chain ran 113 us while every other was done in 20.
struct StarLane {
    int cen, h, k, cl;           // atoms, constraint (-1: a lane past the star's last), cluster
    double cx, cy, cz, hx, hy, hz;  // SHAKE: positions; RATTLE: velocities
    double rx, ry, rz;           // reference (SHAKE) or current (RATTLE) vector, centre - H
    double inv_c, inv_h, wq, dsq;
    double rcp;                  // RATTLE: 1 / wq (0 where wq is not of ordinary size)
    double lam, acc;             // the last multiplier; the total (keep_sum)
    unsigned it;                 // iterations done (alike over the group)
    bool ok;                     // converged in phase 1
};

struct LaneGroup {
    int width, base;
    unsigned mask;
};

__device__ __forceinline__ LaneGroup lane_group(const ClusterArgs &c, int warp) {
    LaneGroup g;
    const int lane = threadIdx.x & 31;
    g.width = c.lane_width[warp];
    g.base = lane & ~(g.width - 1);
    g.mask = ((1u << g.width) - 1u) << g.base;
    return g;
}

// The displacement (or velocity change) of multiplier s.lam, for the groups
// with `run`; every lane of the warp calls.
__device__ __forceinline__ void lane_apply(StarLane &s, const LaneGroup &g, bool run) {
    const unsigned full = 0xffffffffu;
    const double w = s.lam * s.inv_c;
    const double tx = w * s.rx, ty = w * s.ry, tz = w * s.rz;
    // 0.0 - t_0 - t_1 - ..., the first difference as a negation (a lane past
    // the star's last sends 0)
    double ddx, ddy, ddz;
    if (g.width == 1) {
        ddx = -tx; ddy = -ty; ddz = -tz;
    } else {
        ddx = -__shfl_sync(full, tx, g.base);
        ddy = -__shfl_sync(full, ty, g.base);
        ddz = -__shfl_sync(full, tz, g.base);
        for (int q = 1; q < g.width; q++) {
            ddx -= __shfl_sync(full, tx, g.base + q);
            ddy -= __shfl_sync(full, ty, g.base + q);
            ddz -= __shfl_sync(full, tz, g.base + q);
        }
    }
    const double wh = s.lam * s.inv_h;
    const double ux = wh * s.rx, uy = wh * s.ry, uz = wh * s.rz;
    if (run) {
        s.cx += ddx; s.cy += ddy; s.cz += ddz;
        s.hx += ux; s.hy += uy; s.hz += uz;
    }
}

// Jacobi iterations of every group of the warp: phase 1 to the group's own
// convergence (at most `stop`), phase 2 to `stop`.
template <bool RATTLE>
__device__ __forceinline__ void lane_iterate(const ClusterArgs &c, StarLane &s, const LaneGroup &g, unsigned stop,
                                             bool phase1, bool keep_sum) {
    const unsigned full = 0xffffffffu;
    for (;;) {
        const bool run = s.cl >= 0 && s.it < stop && !(phase1 && s.ok);
        if (!__any_sync(full, run)) break;
        double l = 0.0;
        if (s.k >= 0) {
            const double dx = RATTLE ? s.cx - s.hx : cdiff(c, s.cx, s.hx, 0);
            const double dy = RATTLE ? s.cy - s.hy : cdiff(c, s.cy, s.hy, 1);
            const double dz = RATTLE ? s.cz - s.hz : cdiff(c, s.cz, s.hz, 2);
            const double dot = dx * s.rx + dy * s.ry + dz * s.rz;
            if (RATTLE) {
                if (s.rcp != 0.0) l = gm_div_rcp(dot, s.wq, s.rcp);
                else l = s.wq == 0.0 ? 0.0 : dot / s.wq;
            } else {
                const double diff = dx * dx + dy * dy + dz * dz - s.dsq;
                const double denom = s.wq * dot;
                l = (__double_as_longlong(denom) << 1) == 0 ? 0.0 : diff / denom;
            }
        }
        if (run) {
            s.lam = l;
            if (keep_sum) s.acc += l;
        }
        lane_apply(s, g, run);
        // max |lambda| < tol over the group; a NaN counts as 0, as in the
        // sequential sweep's strict comparison
        const unsigned small = __ballot_sync(full, !gm_abs_ge(l, c.tol));
        if (run) {
            s.it++;
            if (phase1) s.ok = (small & g.mask) == g.mask;
        }
    }
}

// The group's lane: atoms and constants.  `v`: the array that the solve
// changes; RATTLE's vectors come from pos, SHAKE's from rvec.
template <bool RATTLE>
__device__ __forceinline__ void lane_constants(const ClusterArgs &c, int warp, StarLane &s) {
    const int4 t = c.lanes[warp * 32 + (threadIdx.x & 31)];
    s.cen = t.x; s.h = t.y; s.k = t.z; s.cl = t.w;
    s.cx = s.cy = s.cz = s.hx = s.hy = s.hz = 0.0;
    s.rx = s.ry = s.rz = s.inv_c = s.inv_h = s.wq = s.dsq = s.rcp = 0.0;
    s.lam = s.acc = 0.0;
    s.it = 0;
    s.ok = false;
    if (s.cl < 0) return;
    s.inv_c = c.inv_mass[s.cen];
    if (s.k >= 0) {
        s.inv_h = c.inv_mass[s.h];
        if (!RATTLE) {
            s.dsq = c.constr_dsq[s.k];
            s.wq = 2.0 * (s.inv_c + s.inv_h);
        }
    }
}
// RATTLE: the bond vector of the fixed positions and (1/m_i + 1/m_j) r^2
__device__ __forceinline__ void lane_bond(const ClusterArgs &c, const double *pos, int n, StarLane &s) {
    if (s.k < 0) return;
    s.rx = cdiff(c, pos[s.cen], pos[s.h], 0);
    s.ry = cdiff(c, pos[n + s.cen], pos[n + s.h], 1);
    s.rz = cdiff(c, pos[2 * n + s.cen], pos[2 * n + s.h], 2);
    const double rsq = s.rx * s.rx + s.ry * s.ry + s.rz * s.rz;
    s.wq = (s.inv_c + s.inv_h) * rsq;
    s.rcp = gm_ordinary(s.wq) ? 1.0 / s.wq : 0.0;
}

// The worst constraint of the group's last iteration (the first in ascending
// order, a NaN never wins), alike over the group.
__device__ __forceinline__ void lane_worst(const StarLane &s, const LaneGroup &g, double &mx, int &worst) {
    const unsigned full = 0xffffffffu;
    const double la = fabs(s.lam) > 0.0 ? fabs(s.lam) : 0.0;
    mx = la;
    for (int o = 1; o < 8; o <<= 1) {
        const double m = __shfl_xor_sync(full, mx, o);
        if (o < g.width) mx = fmax(mx, m);
    }
    const unsigned hit = __ballot_sync(full, s.k >= 0 && la == mx && mx > 0.0) & g.mask;
    worst = __shfl_sync(full, s.k, hit ? __ffs(hit) - 1 : g.base);
}

// After phase 1: the clusters' counts and worst constraints, the failures and
// the largest count (one atomic per warp).
template <bool RATTLE>
__device__ __forceinline__ void lane_report1(const ClusterArgs &c, const StarLane &s, const LaneGroup &g, unsigned *T) {
    double mx;
    int worst;
    lane_worst(s, g, mx, worst);
    const bool leader = s.cl >= 0 && (int)(threadIdx.x & 31) == g.base;
    if (leader) {
        c.cl_iters[s.cl] = (int)s.it;
        c.cl_worst[s.cl] = mx;
        c.cl_worst_idx[s.cl] = worst;
        if (!s.ok) {
            atomicOr(&c.status->error, RATTLE ? (unsigned)GM_DEV_RATTLE_FAIL : (unsigned)GM_DEV_SHAKE_FAIL);
            atomicMin(&c.status->fail_step, c.status->step);
        }
    }
    const unsigned it = __reduce_max_sync(0xffffffffu, leader ? s.it : 0u);
    if ((threadIdx.x & 31) == 0 && it) atomicMax(T, it);
}

// After phase 2 of the groups that iterated (`ran`): counts, worst
// constraints, and the check of the global stop rule.
__device__ __forceinline__ void lane_report2(const ClusterArgs &c, const StarLane &s, const LaneGroup &g, unsigned T,
                                             bool ran) {
    double mx;
    int worst;
    lane_worst(s, g, mx, worst);
    if (ran && s.cl >= 0 && (int)(threadIdx.x & 31) == g.base) {
        c.cl_iters[s.cl] = (int)s.it;
        c.cl_worst[s.cl] = mx;
        c.cl_worst_idx[s.cl] = worst;
        if (!(mx < c.tol) && T < c.max_iter) atomicOr(&c.status->error, (unsigned)GM_DEV_ITER_MISMATCH);
    }
}

template <bool RATTLE>
__device__ void star_phase(const ClusterArgs &c, int warp, double *pos, double *vel, int n, bool phase2) {
    const DevStatus *st = c.status;
    unsigned T = 0;
    if (!phase2) {
        if (st->error) return;
    } else {
        T = RATTLE ? st->rattle_T : st->shake_T;
        if ((st->error & ~(unsigned)(GM_DEV_SHAKE_FAIL | GM_DEV_RATTLE_FAIL)) != 0) return;
    }
    const LaneGroup g = lane_group(c, warp);
    StarLane s;
    lane_constants<RATTLE>(c, warp, s);
    if (phase2) {
        s.it = s.cl >= 0 ? (unsigned)c.cl_iters[s.cl] : T;
        if (!__any_sync(0xffffffffu, s.it < T)) return;
    }
    const bool ran = s.it < T;
    double *v = RATTLE ? vel : pos;
    const int ncst = c.n_constr;
    if (s.cl >= 0) { s.cx = v[s.cen]; s.cy = v[n + s.cen]; s.cz = v[2 * n + s.cen]; }
    if (s.k >= 0) {
        s.hx = v[s.h]; s.hy = v[n + s.h]; s.hz = v[2 * n + s.h];
        if (!RATTLE) {
            // rvec is i - j
            const bool flip = c.constr_i[s.k] != s.cen;
            s.rx = c.rvec[s.k]; s.ry = c.rvec[ncst + s.k]; s.rz = c.rvec[2 * ncst + s.k];
            if (flip) { s.rx = -s.rx; s.ry = -s.ry; s.rz = -s.rz; }
        }
    }
    if (RATTLE) lane_bond(c, pos, n, s);
    const bool keep_sum = !RATTLE && c.lam_sum;
    if (!phase2) {
        if (!RATTLE && c.lam0) {
            if (s.k >= 0) s.acc = s.lam = c.lam0[s.k];
            lane_apply(s, g, s.cl >= 0);
        }
        lane_iterate<RATTLE>(c, s, g, c.max_iter, true, keep_sum);
        lane_report1<RATTLE>(c, s, g, RATTLE ? &c.status->rattle_T : &c.status->shake_T);
    } else {
        if (keep_sum && s.k >= 0) s.acc = c.lam_sum[s.k];
        lane_iterate<RATTLE>(c, s, g, T, false, keep_sum);
        lane_report2(c, s, g, T, ran);
        if (!ran) return;
    }
    if (s.cl >= 0 && (int)(threadIdx.x & 31) == g.base) { v[s.cen] = s.cx; v[n + s.cen] = s.cy; v[2 * n + s.cen] = s.cz; }
    if (s.k >= 0) {
        v[s.h] = s.hx; v[n + s.h] = s.hy; v[2 * n + s.h] = s.hz;
        if (keep_sum) c.lam_sum[s.k] = s.acc;
    }
}

// Clusters of 2-32 constraints on at most 32 atoms (a heavy atom with its H
// atoms): one warp per cluster.  Lane a keeps atom a's coordinates and its
// constraint list in registers, lane q keeps constraint q's bond vector and
// multiplier; values move between lanes by shuffles.  Each lane's arithmetic
// is that of shake_iteration / rattle_iteration in the same order, and the
// largest |lambda| and its constraint (the first in ascending order on ties)
// come from a warp reduction, so the bits are those of the sequential sweep.
constexpr int kWarpRefs = 8;  // constraints per atom handled by the warp path

// Lane a < na adds its atom's displacement over its constraints (ascending,
// from 0.0): every lane runs the loop to the warp's longest list so that
// every shuffle has all 32 lanes.
__device__ __forceinline__ void warp_atom_update(int lane, int na, int nref, int maxref, const int *ref_l,
                                                 const int *ref_s, double im_a, double lam, double rx, double ry,
                                                 double rz, double &X, double &Y, double &Z) {
    double ddx = 0.0, ddy = 0.0, ddz = 0.0;
    for (int r = 0; r < maxref; r++) {
        const bool mine = lane < na && r < nref;
        const int l = mine ? ref_l[r] : 0;
        const double lam_l = __shfl_sync(0xffffffffu, lam, l);
        const double rx_l = __shfl_sync(0xffffffffu, rx, l);
        const double ry_l = __shfl_sync(0xffffffffu, ry, l);
        const double rz_l = __shfl_sync(0xffffffffu, rz, l);
        if (mine) {
            const double w = lam_l * im_a;
            const double tx = w * rx_l, ty = w * ry_l, tz = w * rz_l;
            if (ref_s[r] < 0) { ddx -= tx; ddy -= ty; ddz -= tz; }
            else { ddx += tx; ddy += ty; ddz += tz; }
        }
    }
    if (lane < na) {
        X += ddx;
        Y += ddy;
        Z += ddz;
    }
}

template <bool RATTLE>
__device__ void cluster_warp(const ClusterArgs &c, int cl, double *pos, double *vel, int n, bool phase2) {
    const int lane = threadIdx.x & 31;
    const DevStatus *st = c.status;
    unsigned T = 0;
    if (!phase2) {
        if (st->error) return;
    } else {
        T = RATTLE ? st->rattle_T : st->shake_T;
        if ((st->error & ~(unsigned)(GM_DEV_SHAKE_FAIL | GM_DEV_RATTLE_FAIL)) != 0) return;
        if ((unsigned)c.cl_iters[cl] >= T) return;
    }
    const int c0 = c.cl_cstart[cl], nc = c.cl_cstart[cl + 1] - c0;
    const int a0 = c.cl_astart[cl], na = c.cl_astart[cl + 1] - a0;
    const int ncst = c.n_constr;
    double *v = RATTLE ? vel : pos;
    // atoms: lane a holds atom a and its constraint list (local indices)
    int ag = 0;
    double im_a = 0.0, X = 0.0, Y = 0.0, Z = 0.0;
    int nref = 0, ref_l[kWarpRefs], ref_s[kWarpRefs];
    if (lane < na) {
        ag = c.cl_atoms[a0 + lane];
        im_a = c.inv_mass[ag];
        X = v[ag]; Y = v[n + ag]; Z = v[2 * n + ag];
        const int r0 = c.cl_acstart[a0 + lane], r1 = c.cl_acstart[a0 + lane + 1];
        for (int r = r0; r < r1 && nref < kWarpRefs; r++) {
            const int ref = c.cl_acons[r];
            const int kk = ref >= 0 ? ref : -ref - 1;
            int l = 0;
            for (int t = 0; t < nc; t++) if (c.cl_cons[c0 + t] == kk) l = t;
            ref_l[nref] = l;
            ref_s[nref] = ref >= 0 ? 1 : -1;
            nref++;
        }
    }
    int maxref = nref;
    for (int o = 16; o > 0; o >>= 1) maxref = max(maxref, __shfl_xor_sync(0xffffffffu, maxref, o));
    // constraints: lane q holds constraint q
    int k = 0, il = 0, jl = 0;
    double wq = 0.0, dsq = 0.0, acc = 0.0, rx = 0.0, ry = 0.0, rz = 0.0, lam = 0.0;
    if (lane < nc) {
        k = c.cl_cons[c0 + lane];
        const int i = c.constr_i[k], j = c.constr_j[k];
        for (int t = 0; t < na; t++) {
            const int a = c.cl_atoms[a0 + t];
            if (a == i) il = t;
            if (a == j) jl = t;
        }
        const double inv_mi = c.inv_mass[i], inv_mj = c.inv_mass[j];
        if (!RATTLE) {
            dsq = c.constr_dsq[k];
            rx = c.rvec[k]; ry = c.rvec[ncst + k]; rz = c.rvec[2 * ncst + k];
            wq = 2.0 * (inv_mi + inv_mj);
        } else {
            // constraint.rs:205-215: the bond vector of the fixed positions
            rx = cdiff(c, pos[i], pos[j], 0);
            ry = cdiff(c, pos[n + i], pos[n + j], 1);
            rz = cdiff(c, pos[2 * n + i], pos[2 * n + j], 2);
            const double rsq = rx * rx + ry * ry + rz * rz;
            wq = (inv_mi + inv_mj) * rsq;
        }
    }
    const int k0 = __shfl_sync(0xffffffffu, k, 0);
    const bool keep_sum = !RATTLE && c.lam_sum;
    unsigned it;
    double mx;
    int worst;
    if (!phase2) {
        it = 0;
        mx = 0.0;
        worst = 0;
        if (!RATTLE && c.lam0) {
            if (lane < nc) { acc = c.lam0[k]; lam = acc; }
            warp_atom_update(lane, na, nref, maxref, ref_l, ref_s, im_a, lam, rx, ry, rz, X, Y, Z);
        }
    } else {
        it = (unsigned)c.cl_iters[cl];
        mx = c.cl_worst[cl];
        worst = c.cl_worst_idx[cl];
        if (keep_sum && lane < nc) acc = c.lam_sum[k];
    }
    bool ok = false;
    const unsigned stop = phase2 ? T : c.max_iter;
    while (it < stop) {
        // constraint lanes fetch their two atoms
        const double xi = __shfl_sync(0xffffffffu, X, il), yi = __shfl_sync(0xffffffffu, Y, il),
                     zi = __shfl_sync(0xffffffffu, Z, il);
        const double xj = __shfl_sync(0xffffffffu, X, jl), yj = __shfl_sync(0xffffffffu, Y, jl),
                     zj = __shfl_sync(0xffffffffu, Z, jl);
        double la = 0.0;
        lam = 0.0;
        if (lane < nc) {
            double l_;
            if (RATTLE) {
                const double dvx = xi - xj;
                const double dvy = yi - yj;
                const double dvz = zi - zj;
                const double rel_vel = dvx * rx + dvy * ry + dvz * rz;
                l_ = wq == 0.0 ? 0.0 : rel_vel / wq;
            } else {
                const double dx = cdiff(c, xi, xj, 0);
                const double dy = cdiff(c, yi, yj, 1);
                const double dz = cdiff(c, zi, zj, 2);
                const double diff = dx * dx + dy * dy + dz * dz - dsq;
                const double dot_new_old = dx * rx + dy * ry + dz * rz;
                const double denom = wq * dot_new_old;
                l_ = denom == 0.0 ? 0.0 : diff / denom;
                if (keep_sum) acc += l_;
            }
            la = fabs(l_);
            lam = l_;
        }
        // the largest |lambda| (a NaN never wins, as with the sequential '>')
        // and the first constraint that reaches it
        double m = la > 0.0 ? la : 0.0;
        for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
        const unsigned hit = __ballot_sync(0xffffffffu, lane < nc && la == m && m > 0.0);
        worst = __shfl_sync(0xffffffffu, k, hit ? __ffs(hit) - 1 : 0);
        if (!hit) worst = k0;
        mx = m;
        warp_atom_update(lane, na, nref, maxref, ref_l, ref_s, im_a, lam, rx, ry, rz, X, Y, Z);
        it++;
        if (!phase2 && mx < c.tol) { ok = true; break; }
    }
    if (lane < na) { v[ag] = X; v[n + ag] = Y; v[2 * n + ag] = Z; }
    if (keep_sum && lane < nc) c.lam_sum[k] = acc;
    if (lane == 0) {
        c.cl_iters[cl] = (int)it;
        c.cl_worst[cl] = mx;
        c.cl_worst_idx[cl] = worst;
        if (!phase2) {
            if (!ok) {
                atomicOr(&c.status->error, RATTLE ? (unsigned)GM_DEV_RATTLE_FAIL : (unsigned)GM_DEV_SHAKE_FAIL);
                atomicMin(&c.status->fail_step, c.status->step);
            }
            atomicMax(RATTLE ? &c.status->rattle_T : &c.status->shake_T, it);
        } else if (!(mx < c.tol) && T < c.max_iter) {
            atomicOr(&c.status->error, (unsigned)GM_DEV_ITER_MISMATCH);
        }
    }
}

// Warm start: one displacement with the predicted multipliers lam0, by the
// update of a Jacobi sweep (per-atom deltas over the atom's constraints in
// ascending order from 0.0, then added), before the unchanged iterations.
// The multiplier totals start from lam0.
// Clusters come in three ranges, launched with 32-thread blocks: stars (a
// constraint per lane, n_lane_warps blocks), [n_star_end, n_warp_end) other
// clusters of 2-32 constraints, one per warp; the rest one per thread
// through global memory.
struct ClusterBlocks {
    int star, warp, big;
};

__host__ __device__ __forceinline__ ClusterBlocks cluster_block_ranges(const ClusterArgs &c) {
    ClusterBlocks b;
    b.star = c.n_lane_warps;
    b.warp = c.n_warp_end - c.n_star_end;
    b.big = (c.n_clusters - c.n_warp_end + 31) / 32;
    return b;
}

int cluster_blocks(const ClusterArgs &c) {
    const ClusterBlocks b = cluster_block_ranges(c);
    return b.star + b.warp + b.big;
}

// Runs the cluster of this thread (or warp) by its class; false for the
// global-memory class, which the caller handles, with *cl set.
template <bool RATTLE>
__device__ __forceinline__ bool cluster_dispatch(const ClusterArgs &c, double *pos, double *vel, int n, bool phase2,
                                                 int *cl) {
    const ClusterBlocks b = cluster_block_ranges(c);
    int blk = blockIdx.x;
    if (blk < b.star) {
        star_phase<RATTLE>(c, blk, pos, vel, n, phase2);
        return true;
    }
    blk -= b.star;
    if (blk < b.warp) {
        cluster_warp<RATTLE>(c, c.n_star_end + blk, pos, vel, n, phase2);
        return true;
    }
    blk -= b.warp;
    *cl = c.n_warp_end + blk * 32 + threadIdx.x;
    return false;
}

__global__ void warm_start_apply(ClusterArgs c, double *pos, int n_atoms) {
    // big clusters only: the other paths apply the warm start themselves
    const ClusterBlocks b = cluster_block_ranges(c);
    const int blk = (int)blockIdx.x - b.star - b.warp;
    if (blk < 0) return;
    const int cl = c.n_warp_end + blk * 32 + threadIdx.x;
    if (cl >= c.n_clusters || c.status->error) return;
    const int nc = c.n_constr;
    if (c.lam_sum)
        for (int q = c.cl_cstart[cl]; q < c.cl_cstart[cl + 1]; q++) c.lam_sum[c.cl_cons[q]] = c.lam0[c.cl_cons[q]];
    for (int q = c.cl_astart[cl]; q < c.cl_astart[cl + 1]; q++) {
        const int a = c.cl_atoms[q];
        const double inv_m = c.inv_mass[a];
        double ddx = 0.0, ddy = 0.0, ddz = 0.0;
        for (int r = c.cl_acstart[q]; r < c.cl_acstart[q + 1]; r++) {
            const int ref = c.cl_acons[r];
            const int k = ref >= 0 ? ref : -ref - 1;
            const double w = c.lam0[k] * inv_m;
            const double tx = w * c.rvec[k], ty = w * c.rvec[nc + k], tz = w * c.rvec[2 * nc + k];
            if (ref < 0) { ddx -= tx; ddy -= ty; ddz -= tz; }
            else { ddx += tx; ddy += ty; ddz += tz; }
        }
        pos[a] += ddx;
        pos[n_atoms + a] += ddy;
        pos[2 * n_atoms + a] += ddz;
    }
}

template <bool RATTLE>
__global__ void cluster_phase1(ClusterArgs c, double *pos, double *vel, int n_atoms) {
    int cl = 0;
    if (cluster_dispatch<RATTLE>(c, pos, vel, n_atoms, false, &cl)) return;
    if (cl >= c.n_clusters) return;
    if (c.status->error) return;
    double mx = 0.0;
    int worst = 0;
    unsigned it = 0;
    bool ok = false;
    while (it < c.max_iter) {
        if (RATTLE) rattle_iteration(c, cl, pos, vel, n_atoms, mx, worst);
        else shake_iteration(c, cl, c.rvec, pos, n_atoms, mx, worst);
        it++;
        if (mx < c.tol) { ok = true; break; }
    }
    c.cl_iters[cl] = (int)it;
    c.cl_worst[cl] = mx;
    c.cl_worst_idx[cl] = worst;
    if (!ok) {
        atomicOr(&c.status->error, RATTLE ? (unsigned)GM_DEV_RATTLE_FAIL : (unsigned)GM_DEV_SHAKE_FAIL);
        atomicMin(&c.status->fail_step, c.status->step);
    }
    atomicMax(RATTLE ? &c.status->rattle_T : &c.status->shake_T, it);
}

template <bool RATTLE>
__global__ void cluster_phase2(ClusterArgs c, double *pos, double *vel, int n_atoms) {
    int cl = 0;
    if (cluster_dispatch<RATTLE>(c, pos, vel, n_atoms, true, &cl)) return;
    if (cl >= c.n_clusters) return;
    const unsigned T = RATTLE ? c.status->rattle_T : c.status->shake_T;
    if ((c.status->error & ~(unsigned)(GM_DEV_SHAKE_FAIL | GM_DEV_RATTLE_FAIL)) != 0) return;
    unsigned it = (unsigned)c.cl_iters[cl];
    if (it >= T) return;
    double mx = c.cl_worst[cl];
    int worst = c.cl_worst_idx[cl];
    while (it < T) {
        if (RATTLE) rattle_iteration(c, cl, pos, vel, n_atoms, mx, worst);
        else shake_iteration(c, cl, c.rvec, pos, n_atoms, mx, worst);
        it++;
    }
    c.cl_iters[cl] = (int)it;
    c.cl_worst[cl] = mx;
    c.cl_worst_idx[cl] = worst;
    // the global stop at T needs every cluster below tol at iteration T
    if (!(mx < c.tol) && T < c.max_iter) atomicOr(&c.status->error, (unsigned)GM_DEV_ITER_MISMATCH);
}

// ---- the constrained step in two cooperative launches --------------------
//
// Every constraint has a lane (star clusters only), every atom of no
// constraint a thread.  The separate kernels (half-kick, drift, reference
// vectors, two phases, resync, check, pack; half-kick, two phases, step
// count: 14 launches) each cost 2 to 5 us of launch, load and drain for a few
// hundred nanoseconds of work; here the state stays in registers from the kick
// to the pack, and the two phases of a solve meet at one grid barrier.  The
// operations and their order are those of the separate kernels, which remain
// for the trait's calls, the warm start and other cluster classes.
// 20 steps of 1,536 atoms of water 3151 -> 2901 us, 10 steps of 24,000 with
// frames 3852 -> 3645 us, 5 steps of the 20,011-atom chain 1193 -> 1090 us (with
// the WHILE graph and the quads below 2123, 3465 and 1062).

__device__ __forceinline__ double kicked(double v, long long force, double inv_m, double dt_half) {
    const double f = (double)force * GM_FIX_INV;
    return v + dt_half * f * inv_m * kForceToAccel;
}

// Position of atom i after its drift: pack, cleared forces, rebuild check.
__device__ __forceinline__ void finish_atom(const SolveStepArgs &sa, const PackArgs &pk, int i, double x, double y,
                                            double z, int &need, int &bad) {
    const int n = sa.n, sl = pk.slot_of[i], sy = sa.atom_sys[i];
    const GridInfo *g = pk.grid + sy;
    gm_pack_record(pk.coord + 2 * sl, x - g->origin[0], y - g->origin[1], z - g->origin[2], pk.qw[i]);
    if (pk.fp64) {
        pk.pos64s[sl] = make_double4(x, y, z, pk.charge64[i]);
        pk.type_sorted[sl] = pk.type[i];
    }
    for (int d = 0; d < 3; d++) sa.force[d * n + i] = 0;
    bad |= !(isfinite(x) && isfinite(y) && isfinite(z));
    const double dx = x - sa.ref[i], dy = y - sa.ref[n + i], dz = z - sa.ref[2 * n + i];
    const double d2 = dx * dx + dy * dy + dz * dz;
    if (gm_moved_far(d2, sa.far_sq)) sa.sys_far[sy] = 1u;
    if (d2 > sa.thr_sq) {
        sa.sys_flag[sy] = 1u;
        need = 1;
    }
}

// The last block of the launch to get here (its thread 0 alone).
__device__ __forceinline__ bool last_block(DevStatus *st) {
    __threadfence();
    if (atomicAdd(&st->blocks_done, 1u) != gridDim.x - 1) return false;
    __threadfence();
    st->blocks_done = 0;
    return true;
}

// Phase 1's outcome of a warp of stars: the largest count and the failures
// (kept in the solve's own words: the error word must not change before every
// block has read it).
template <bool RATTLE>
__device__ __forceinline__ void lane_report_step(const ClusterArgs &c, const StarLane &s, const LaneGroup &g,
                                                 SolveSync *sy) {
    double mx;
    int worst;
    lane_worst(s, g, mx, worst);
    const bool leader = s.cl >= 0 && (int)(threadIdx.x & 31) == g.base;
    if (leader) {
        c.cl_iters[s.cl] = (int)s.it;
        c.cl_worst[s.cl] = mx;
        c.cl_worst_idx[s.cl] = worst;
        if (!s.ok) {
            atomicOr(&sy->fail, 1u);
            atomicMin(&c.status->fail_step, c.status->step);
        }
    }
    const unsigned it = __reduce_max_sync(0xffffffffu, leader ? s.it : 0u);
    if ((threadIdx.x & 31) == 0 && it) atomicMax(&sy->T, it);
}

// The first of a thread's atoms of no constraint: the threads past the `lanes`
// solver lanes take them first.
__device__ __forceinline__ int first_free(int tid, int threads, int lanes) {
    return tid >= lanes ? tid - lanes : tid + threads - lanes;
}

// Kick, drift and what follows it for the atoms of no constraint; the kicked
// velocity goes to dref for the case of a failed projection, which skips the
// resync.
__device__ __forceinline__ void free_drift(const ClusterArgs &c, const SolveStepArgs &sa, const PackArgs &pk, bool err0,
                                           int free0, int threads, int &need, int &bad) {
    const int n = sa.n;
    for (int q = free0; q < sa.n_free; q += threads) {
        const int i = sa.free_atoms[q];
        double np[3];
        const double inv_m = c.inv_mass[i];
        for (int d = 0; d < 3; d++) {
            const double p = sa.pos[d * n + i];
            np[d] = p;
            if (!err0) {
                const double v = kicked(sa.vel[d * n + i], sa.force[d * n + i], inv_m, sa.dt_half);
                np[d] = p + sa.dt * v;
                sa.pos[d * n + i] = np[d];
                sa.dref[d * n + i] = v;
                sa.vel[d * n + i] = gm_div_by_dt(np[d] - p, sa.dt, sa.inv_dt);
            }
        }
        finish_atom(sa, pk, i, np[0], np[1], np[2], need, bad);
    }
}
__device__ __forceinline__ void free_kicked(const SolveStepArgs &sa, int free0, int threads) {
    const int n = sa.n;
    for (int q = free0; q < sa.n_free; q += threads) {
        const int i = sa.free_atoms[q];
        for (int d = 0; d < 3; d++) sa.vel[d * n + i] = sa.dref[d * n + i];
    }
}
__device__ __forceinline__ void free_kick(const ClusterArgs &c, const SolveStepArgs &sa, int free0, int threads) {
    const int n = sa.n;
    for (int q = free0; q < sa.n_free; q += threads) {
        const int i = sa.free_atoms[q];
        const double inv_m = c.inv_mass[i];
        for (int d = 0; d < 3; d++) sa.vel[d * n + i] = kicked(sa.vel[d * n + i], sa.force[d * n + i], inv_m, sa.dt_half);
    }
}

// The WHILE node round the step ends unless RATTLE's bookkeeping asks for
// another step (a barrier that times out, in either launch, skips that).
__device__ __forceinline__ void loop_off(const SolveStepArgs &sa) {
    if (sa.loop && blockIdx.x == 0 && threadIdx.x == 0)
        cudaGraphSetConditional((cudaGraphConditionalHandle)sa.loop, 0u);
}

// The ends of the two kernels: the last block's bookkeeping.
__device__ __forceinline__ void shake_tail(const SolveStepArgs &sa, DevStatus *st, unsigned T, bool fail, int need,
                                           int bad) {
    SolveSync *sy = sa.sync;
    need = __syncthreads_or(need);
    bad = __syncthreads_or(bad);
    if (threadIdx.x == 0) {
        if (need) atomicOr(&st->rebuild, 1u);
        if (bad) atomicOr(&st->error, (unsigned)GM_DEV_NONFINITE_POS);
        if (last_block(st)) {
            st->shake_T = T;
            if (fail) atomicOr(&st->error, (unsigned)GM_DEV_SHAKE_FAIL);
            sy->T = 0;
            sy->fail = 0;
            const unsigned r = atomicOr(&st->rebuild, 0u), e = atomicOr(&st->error, 0u);
            if (sa.cond) cudaGraphSetConditional((cudaGraphConditionalHandle)sa.cond, (r && !e) ? 1u : 0u);
        }
    }
}

__device__ __forceinline__ void rattle_tail(const SolveStepArgs &sa, DevStatus *st, unsigned T, bool fail) {
    SolveSync *sy = sa.sync;
    __syncthreads();
    if (threadIdx.x == 0 && last_block(st)) {
        st->rattle_T = T;
        if (fail) atomicOr(&st->error, (unsigned)GM_DEV_RATTLE_FAIL);
        sy->T = 0;
        sy->fail = 0;
        if (atomicOr(&st->error, 0u) == 0) {  // step_kernel's count
            st->step += 1;
            if (st->shake_T || T) {
                st->c_steps += 1;
                st->shake_sum += st->shake_T;
                st->rattle_sum += T;
            }
            if (sa.loop) {
                const long long left = sy->todo - 1;
                sy->todo = left;
                cudaGraphSetConditional((cudaGraphConditionalHandle)sa.loop, left > 0 ? 1u : 0u);
            }
        }
    }
}

__global__ void __launch_bounds__(128) shake_step_kernel(ClusterArgs c, SolveStepArgs sa, PackArgs pk) {
    DevStatus *st = c.status;
    SolveSync *sy = sa.sync;
    const int n = sa.n, tid = blockIdx.x * blockDim.x + threadIdx.x, warp = tid >> 5;
    const bool err0 = gm_ld_acquire(&st->error) != 0;  // before any block may change it (the barrier)
    loop_off(sa);
    const bool lanes = warp < c.n_lane_warps;            // warp-uniform
    int need = 0, bad = 0;
    StarLane s;
    LaneGroup g;
    double pc[3], vc[3], ph[3], vh[3];  // before the drift; after the kick
    s.cl = s.k = -1;
    if (lanes) {
        g = lane_group(c, warp);
        lane_constants<false>(c, warp, s);
        if (s.cl >= 0) {
            for (int d = 0; d < 3; d++) {
                pc[d] = sa.pos[d * n + s.cen];
                vc[d] = sa.vel[d * n + s.cen];
                if (!err0) vc[d] = kicked(vc[d], sa.force[d * n + s.cen], s.inv_c, sa.dt_half);
            }
        }
        if (s.k >= 0) {
            for (int d = 0; d < 3; d++) {
                ph[d] = sa.pos[d * n + s.h];
                vh[d] = sa.vel[d * n + s.h];
                if (!err0) vh[d] = kicked(vh[d], sa.force[d * n + s.h], s.inv_h, sa.dt_half);
            }
        }
        if (!err0) {
            if (s.cl >= 0) { s.cx = pc[0] + sa.dt * vc[0]; s.cy = pc[1] + sa.dt * vc[1]; s.cz = pc[2] + sa.dt * vc[2]; }
            if (s.k >= 0) {
                s.hx = ph[0] + sa.dt * vh[0]; s.hy = ph[1] + sa.dt * vh[1]; s.hz = ph[2] + sa.dt * vh[2];
                s.rx = cdiff(c, pc[0], ph[0], 0);
                s.ry = cdiff(c, pc[1], ph[1], 1);
                s.rz = cdiff(c, pc[2], ph[2], 2);
            }
            lane_iterate<false>(c, s, g, c.max_iter, true, false);
            lane_report_step<false>(c, s, g, sy);
        }
    }
    const int threads = gridDim.x * blockDim.x, free0 = first_free(tid, threads, c.n_lane_warps * 32);
    free_drift(c, sa, pk, err0, free0, threads, need, bad);
    if (!gm_grid_barrier(&sy->arrive, &sy->gen, st)) return;
    const unsigned T = gm_ld_acquire(&sy->T);
    const bool fail = gm_ld_acquire(&sy->fail) != 0;
    if (lanes) {
        if (!err0) {
            const bool ran = s.cl >= 0 && s.it < T;
            lane_iterate<false>(c, s, g, T, false, false);
            lane_report2(c, s, g, T, ran);
        } else {
            s.cx = pc[0]; s.cy = pc[1]; s.cz = pc[2];
            s.hx = ph[0]; s.hy = ph[1]; s.hz = ph[2];
        }
        const bool leader = s.cl >= 0 && (int)(threadIdx.x & 31) == g.base;
        if (leader) {
            if (!err0) {
                const double x[3] = {s.cx, s.cy, s.cz};
                for (int d = 0; d < 3; d++) {
                    sa.pos[d * n + s.cen] = x[d];
                    sa.vel[d * n + s.cen] = fail ? vc[d] : gm_div_by_dt(x[d] - pc[d], sa.dt, sa.inv_dt);
                }
            }
            finish_atom(sa, pk, s.cen, s.cx, s.cy, s.cz, need, bad);
        }
        if (s.k >= 0) {
            if (!err0) {
                const double x[3] = {s.hx, s.hy, s.hz};
                for (int d = 0; d < 3; d++) {
                    sa.pos[d * n + s.h] = x[d];
                    sa.vel[d * n + s.h] = fail ? vh[d] : gm_div_by_dt(x[d] - ph[d], sa.dt, sa.inv_dt);
                }
            }
            finish_atom(sa, pk, s.h, s.hx, s.hy, s.hz, need, bad);
        }
    }
    if (!err0 && fail) free_kicked(sa, free0, threads);
    shake_tail(sa, st, T, fail, need, bad);
}

__global__ void __launch_bounds__(128) rattle_step_kernel(ClusterArgs c, SolveStepArgs sa) {
    DevStatus *st = c.status;
    SolveSync *sy = sa.sync;
    const int n = sa.n, tid = blockIdx.x * blockDim.x + threadIdx.x, warp = tid >> 5;
    const bool err0 = gm_ld_acquire(&st->error) != 0;
    const bool lanes = warp < c.n_lane_warps;
    StarLane s;
    LaneGroup g;
    if (lanes && !err0) {
        g = lane_group(c, warp);
        lane_constants<true>(c, warp, s);
        if (s.cl >= 0) {
            s.cx = kicked(sa.vel[s.cen], sa.force[s.cen], s.inv_c, sa.dt_half);
            s.cy = kicked(sa.vel[n + s.cen], sa.force[n + s.cen], s.inv_c, sa.dt_half);
            s.cz = kicked(sa.vel[2 * n + s.cen], sa.force[2 * n + s.cen], s.inv_c, sa.dt_half);
        }
        if (s.k >= 0) {
            s.hx = kicked(sa.vel[s.h], sa.force[s.h], s.inv_h, sa.dt_half);
            s.hy = kicked(sa.vel[n + s.h], sa.force[n + s.h], s.inv_h, sa.dt_half);
            s.hz = kicked(sa.vel[2 * n + s.h], sa.force[2 * n + s.h], s.inv_h, sa.dt_half);
        }
        lane_bond(c, sa.pos, n, s);
        lane_iterate<true>(c, s, g, c.max_iter, true, false);
        lane_report_step<true>(c, s, g, sy);
    }
    const int threads = gridDim.x * blockDim.x;
    if (!err0) free_kick(c, sa, first_free(tid, threads, c.n_lane_warps * 32), threads);
    if (!gm_grid_barrier(&sy->arrive, &sy->gen, st)) return;
    const unsigned T = gm_ld_acquire(&sy->T);
    const bool fail = gm_ld_acquire(&sy->fail) != 0;
    if (lanes && !err0) {
        const bool ran = s.cl >= 0 && s.it < T;
        lane_iterate<true>(c, s, g, T, false, false);
        lane_report2(c, s, g, T, ran);
        if (s.cl >= 0 && (int)(threadIdx.x & 31) == g.base) {
            sa.vel[s.cen] = s.cx; sa.vel[n + s.cen] = s.cy; sa.vel[2 * n + s.cen] = s.cz;
        }
        if (s.k >= 0) { sa.vel[s.h] = s.hx; sa.vel[n + s.h] = s.hy; sa.vel[2 * n + s.h] = s.hz; }
    }
    rattle_tail(sa, st, T, fail);
}

// ---- the same step with four lanes a constraint ---------------------------
//
// For systems whose lanes leave schedulers without a warp: lane d of a quad
// holds component d of the centre, the H atom and the vector (the fourth lane
// repeats z and stores nothing), so a difference, a product or an update of
// three components is one FP64 instruction of the warp instead of three; the
// sums over components take the three products by shuffles and add them in the
// order of the lane per constraint.  An iteration of a two-H star is about 28
// FP64 instructions in a row against 43 (SHAKE) and 14 against 28 (RATTLE); the
// two kernels at 1,536 atoms of water 37 -> 26 and 39 -> 28 us.
struct CompLane {
    int cen, h, k, cl, d;    // atoms, constraint, cluster (as in StarLane); component
    double x, y, r;          // centre, H atom (SHAKE: positions, RATTLE: velocities); the vector
    double inv_c, inv_h, wq, dsq, rcp, lam, box;
    unsigned it;
    bool ok;
};

__device__ __forceinline__ double comp_dot(double p) {  // over the quad, every lane of the warp calls
    const unsigned full = 0xffffffffu;
    const double p0 = __shfl_sync(full, p, 0, 4), p1 = __shfl_sync(full, p, 1, 4), p2 = __shfl_sync(full, p, 2, 4);
    return p0 + p1 + p2;
}
__device__ __forceinline__ double comp_diff(const ClusterArgs &c, const CompLane &s, double a, double b) {
    const double v = a - b;
    return c.mi ? gm_min_image(v, s.box) : v;
}

// The quad's constraint and constants; the group in lanes of the warp.
template <bool RATTLE>
__device__ __forceinline__ LaneGroup comp_init(const ClusterArgs &c, int warp, CompLane &s) {
    const int lane = threadIdx.x & 31, q = warp * 8 + (lane >> 2);
    LaneGroup g;
    g.width = 4 * c.lane_width[q >> 5];
    g.base = lane & ~(g.width - 1);
    g.mask = g.width == 32 ? 0xffffffffu : ((1u << g.width) - 1u) << g.base;
    const int4 t = c.lanes[q];
    s.cen = t.x; s.h = t.y; s.k = t.z; s.cl = t.w;
    s.d = min(lane & 3, 2);
    s.box = s.d == 0 ? c.box64[0] : s.d == 1 ? c.box64[1] : c.box64[2];
    s.x = s.y = s.r = s.inv_c = s.inv_h = s.wq = s.dsq = s.rcp = s.lam = 0.0;
    s.it = 0;
    s.ok = false;
    if (s.cl >= 0) s.inv_c = c.inv_mass[s.cen];
    if (s.k >= 0) {
        s.inv_h = c.inv_mass[s.h];
        if (!RATTLE) {
            s.dsq = c.constr_dsq[s.k];
            s.wq = 2.0 * (s.inv_c + s.inv_h);
        }
    }
    return g;
}

// lane_iterate and lane_apply, a component per lane
template <bool RATTLE>
__device__ __forceinline__ void comp_iterate(const ClusterArgs &c, CompLane &s, const LaneGroup &g, unsigned stop,
                                             bool phase1) {
    const unsigned full = 0xffffffffu;
    const int sub = threadIdx.x & 3;
    for (;;) {
        const bool run = s.cl >= 0 && s.it < stop && !(phase1 && s.ok);
        if (!__any_sync(full, run)) break;
        double l = 0.0;
        const double dx = RATTLE ? s.x - s.y : comp_diff(c, s, s.x, s.y);
        const double dot = comp_dot(dx * s.r);
        if (RATTLE) {
            if (s.k >= 0) {
                if (s.rcp != 0.0) l = gm_div_rcp(dot, s.wq, s.rcp);
                else l = s.wq == 0.0 ? 0.0 : dot / s.wq;
            }
        } else {
            const double diff = comp_dot(dx * dx) - s.dsq;
            if (s.k >= 0) {
                const double denom = s.wq * dot;
                l = (__double_as_longlong(denom) << 1) == 0 ? 0.0 : diff / denom;
            }
        }
        if (run) s.lam = l;
        const double w = s.lam * s.inv_c;
        const double t = w * s.r;
        double dd = -__shfl_sync(full, t, g.base + sub);
        for (int q = 4; q < g.width; q += 4) dd -= __shfl_sync(full, t, g.base + q + sub);
        const double wh = s.lam * s.inv_h;
        const double u = wh * s.r;
        if (run) {
            s.x += dd;
            s.y += u;
        }
        const unsigned small = __ballot_sync(full, !gm_abs_ge(l, c.tol));
        if (run) {
            s.it++;
            if (phase1) s.ok = (small & g.mask) == g.mask;
        }
    }
}

// lane_worst, lane_report_step and lane_report2 over quads
__device__ __forceinline__ void comp_worst(const CompLane &s, const LaneGroup &g, double &mx, int &worst) {
    const unsigned full = 0xffffffffu;
    const double la = fabs(s.lam) > 0.0 ? fabs(s.lam) : 0.0;
    mx = la;
    for (int o = 4; o < 32; o <<= 1) {
        const double m = __shfl_xor_sync(full, mx, o);
        if (o < g.width) mx = fmax(mx, m);
    }
    const unsigned hit = __ballot_sync(full, s.k >= 0 && la == mx && mx > 0.0) & g.mask;
    worst = __shfl_sync(full, s.k, hit ? __ffs(hit) - 1 : g.base);
}
__device__ __forceinline__ void comp_report_step(const ClusterArgs &c, const CompLane &s, const LaneGroup &g,
                                                 SolveSync *sy) {
    double mx;
    int worst;
    comp_worst(s, g, mx, worst);
    const bool leader = s.cl >= 0 && (int)(threadIdx.x & 31) == g.base;
    if (leader) {
        c.cl_iters[s.cl] = (int)s.it;
        c.cl_worst[s.cl] = mx;
        c.cl_worst_idx[s.cl] = worst;
        if (!s.ok) {
            atomicOr(&sy->fail, 1u);
            atomicMin(&c.status->fail_step, c.status->step);
        }
    }
    const unsigned it = __reduce_max_sync(0xffffffffu, leader ? s.it : 0u);
    if ((threadIdx.x & 31) == 0 && it) atomicMax(&sy->T, it);
}
__device__ __forceinline__ void comp_report2(const ClusterArgs &c, const CompLane &s, const LaneGroup &g, unsigned T,
                                             bool ran) {
    double mx;
    int worst;
    comp_worst(s, g, mx, worst);
    if (ran && s.cl >= 0 && (int)(threadIdx.x & 31) == g.base) {
        c.cl_iters[s.cl] = (int)s.it;
        c.cl_worst[s.cl] = mx;
        c.cl_worst_idx[s.cl] = worst;
        if (!(mx < c.tol) && T < c.max_iter) atomicOr(&c.status->error, (unsigned)GM_DEV_ITER_MISMATCH);
    }
}

// finish_atom by a quad (with `on`): a component a lane, the fourth the charge;
// every lane of the warp calls.
__device__ __forceinline__ void comp_finish(const SolveStepArgs &sa, const PackArgs &pk, bool on, int i, int d, double x,
                                            int &need, int &bad) {
    const int n = sa.n, sub = threadIdx.x & 3;
    int sy = 0;
    double dx = 0.0;
    if (on) {
        const int sl = pk.slot_of[i];
        sy = sa.atom_sys[i];
        float *rec = reinterpret_cast<float *>(pk.coord + 2 * sl);
        if (sub < 3) {
            gm_pack_component(rec + sub, x - pk.grid[sy].origin[d]);
            sa.force[d * n + i] = 0;
            bad |= !isfinite(x);
            dx = x - sa.ref[d * n + i];
        } else {
            const float2 qw = pk.qw[i];
            rec[3] = qw.x;
            rec[7] = qw.y;
        }
        if (pk.fp64) {
            reinterpret_cast<double *>(pk.pos64s + sl)[sub] = sub < 3 ? x : pk.charge64[i];
            if (sub == 3) pk.type_sorted[sl] = pk.type[i];
        }
    }
    const double d2 = comp_dot(dx * dx);
    if (on) {
        if (gm_moved_far(d2, sa.far_sq)) sa.sys_far[sy] = 1u;
        if (d2 > sa.thr_sq) {
            sa.sys_flag[sy] = 1u;
            need = 1;
        }
    }
}

__global__ void __launch_bounds__(32) shake_comp_kernel(ClusterArgs c, SolveStepArgs sa, PackArgs pk) {
    DevStatus *st = c.status;
    SolveSync *sy = sa.sync;
    const int n = sa.n, tid = blockIdx.x * blockDim.x + threadIdx.x, warp = tid >> 5, sub = tid & 3;
    const bool err0 = gm_ld_acquire(&st->error) != 0;
    const bool lanes = warp < 4 * c.n_lane_warps;
    int need = 0, bad = 0;
    loop_off(sa);
    CompLane s;
    LaneGroup g;
    double pc = 0.0, vc = 0.0, ph = 0.0, vh = 0.0;  // before the drift; after the kick
    if (lanes) {
        g = comp_init<false>(c, warp, s);
        if (s.cl >= 0) {
            const int q = s.d * n + s.cen;
            pc = sa.pos[q];
            vc = sa.vel[q];
            if (!err0) vc = kicked(vc, sa.force[q], s.inv_c, sa.dt_half);
        }
        if (s.k >= 0) {
            const int q = s.d * n + s.h;
            ph = sa.pos[q];
            vh = sa.vel[q];
            if (!err0) vh = kicked(vh, sa.force[q], s.inv_h, sa.dt_half);
        }
        if (!err0) {
            if (s.cl >= 0) s.x = pc + sa.dt * vc;
            if (s.k >= 0) {
                s.y = ph + sa.dt * vh;
                s.r = comp_diff(c, s, pc, ph);
            }
            comp_iterate<false>(c, s, g, c.max_iter, true);
            comp_report_step(c, s, g, sy);
        }
    }
    const int threads = gridDim.x * blockDim.x, free0 = first_free(tid, threads, c.n_lane_warps * 128);
    free_drift(c, sa, pk, err0, free0, threads, need, bad);
    if (!gm_grid_barrier(&sy->arrive, &sy->gen, st)) return;
    const unsigned T = gm_ld_acquire(&sy->T);
    const bool fail = gm_ld_acquire(&sy->fail) != 0;
    if (lanes) {
        if (!err0) {
            const bool ran = s.cl >= 0 && s.it < T;
            comp_iterate<false>(c, s, g, T, false);
            comp_report2(c, s, g, T, ran);
        } else {
            s.x = pc;
            s.y = ph;
        }
        const bool leader = s.cl >= 0 && (int)(threadIdx.x & 28) == g.base;
        if (leader && !err0 && sub < 3) {
            sa.pos[s.d * n + s.cen] = s.x;
            sa.vel[s.d * n + s.cen] = fail ? vc : gm_div_by_dt(s.x - pc, sa.dt, sa.inv_dt);
        }
        comp_finish(sa, pk, leader, s.cen, s.d, s.x, need, bad);
        if (s.k >= 0 && !err0 && sub < 3) {
            sa.pos[s.d * n + s.h] = s.y;
            sa.vel[s.d * n + s.h] = fail ? vh : gm_div_by_dt(s.y - ph, sa.dt, sa.inv_dt);
        }
        comp_finish(sa, pk, s.k >= 0, s.h, s.d, s.y, need, bad);
    }
    if (!err0 && fail) free_kicked(sa, free0, threads);
    shake_tail(sa, st, T, fail, need, bad);
}

__global__ void __launch_bounds__(32) rattle_comp_kernel(ClusterArgs c, SolveStepArgs sa) {
    DevStatus *st = c.status;
    SolveSync *sy = sa.sync;
    const int n = sa.n, tid = blockIdx.x * blockDim.x + threadIdx.x, warp = tid >> 5, sub = tid & 3;
    const bool err0 = gm_ld_acquire(&st->error) != 0;
    const bool lanes = warp < 4 * c.n_lane_warps;
    CompLane s;
    LaneGroup g;
    if (lanes && !err0) {
        g = comp_init<true>(c, warp, s);
        double pc = 0.0, ph = 0.0;
        if (s.cl >= 0) {
            const int q = s.d * n + s.cen;
            s.x = kicked(sa.vel[q], sa.force[q], s.inv_c, sa.dt_half);
            pc = sa.pos[q];
        }
        if (s.k >= 0) {
            const int q = s.d * n + s.h;
            s.y = kicked(sa.vel[q], sa.force[q], s.inv_h, sa.dt_half);
            ph = sa.pos[q];
            s.r = comp_diff(c, s, pc, ph);
        }
        // lane_bond
        const double rsq = comp_dot(s.r * s.r);
        if (s.k >= 0) {
            s.wq = (s.inv_c + s.inv_h) * rsq;
            s.rcp = gm_ordinary(s.wq) ? 1.0 / s.wq : 0.0;
        }
        comp_iterate<true>(c, s, g, c.max_iter, true);
        comp_report_step(c, s, g, sy);
    }
    const int threads = gridDim.x * blockDim.x;
    if (!err0) free_kick(c, sa, first_free(tid, threads, c.n_lane_warps * 128), threads);
    if (!gm_grid_barrier(&sy->arrive, &sy->gen, st)) return;
    const unsigned T = gm_ld_acquire(&sy->T);
    const bool fail = gm_ld_acquire(&sy->fail) != 0;
    if (lanes && !err0) {
        const bool ran = s.cl >= 0 && s.it < T;
        comp_iterate<true>(c, s, g, T, false);
        comp_report2(c, s, g, T, ran);
        if (s.cl >= 0 && (int)(threadIdx.x & 28) == g.base && sub < 3) sa.vel[s.d * n + s.cen] = s.x;
        if (s.k >= 0 && sub < 3) sa.vel[s.d * n + s.h] = s.y;
    }
    rattle_tail(sa, st, T, fail);
}

__global__ void solve_begin_kernel(SolveSync *two, long long todo) {
    SolveSync z{};
    two[0] = z;
    z.todo = todo;
    two[1] = z;
}

__global__ void reset_T(DevStatus *st, int rattle) {
    if (rattle) st->rattle_T = 0; else st->shake_T = 0;
}

__global__ void step_kernel(DevStatus *st) {
    if (st->error) return;
    st->step += 1;
    if (st->shake_T || st->rattle_T) {
        st->c_steps += 1;
        st->shake_sum += st->shake_T;
        st->rattle_sum += st->rattle_T;
    }
}

__global__ void kinetic_partial(int n, const double *vel, const double *mass, double *partial) {
    __shared__ double s[256];
    double acc = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const double vx = vel[i], vy = vel[n + i], vz = vel[2 * n + i];
        acc += mass[i] * (vx * vx + vy * vy + vz * vz);
    }
    s[threadIdx.x] = acc;
    __syncthreads();
    for (int k = 128; k > 0; k >>= 1) {
        if (threadIdx.x < k) s[threadIdx.x] += s[threadIdx.x + k];
        __syncthreads();
    }
    if (threadIdx.x == 0) partial[blockIdx.x] = s[0];
}

// Trajectory frame (see gm_launch_frame).  The completed step count is the
// counter plus one while the unconstrained step's closing half-kick is still
// pending; every block takes the same early exit.
__global__ void __launch_bounds__(256) frame_kernel(int n, const double *pos, const double *vel,
                                                    const long long *force, const double *inv_mass,
                                                    const double *mass, double dt_half, DevStatus *st, FrameArgs f) {
    const bool tail = st->tail_pending != 0;
    const unsigned long long step = st->step + (tail ? 1ull : 0ull);
    if (st->error || f.interval <= 0 || step % (unsigned long long)f.interval != 0) return;
    const unsigned slot = st->frame_n;  // every block reads it before the last block advances it
    const bool store = slot < (unsigned)f.cap;
    float *fx = f.xyz + (size_t)(store ? slot : 0) * 3 * (size_t)n;
    __shared__ double s[256];
    __shared__ bool last;
    double acc = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double v[3];
        for (int d = 0; d < 3; d++) {
            if (store) fx[(size_t)d * n + i] = (float)pos[d * n + i];
            v[d] = vel[d * n + i];
            if (tail) {
                const double fd = (double)force[d * n + i] * GM_FIX_INV;
                v[d] += dt_half * fd * inv_mass[i] * kForceToAccel;
            }
        }
        acc += mass[i] * (v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);  // kinetic_partial's order
    }
    s[threadIdx.x] = acc;
    __syncthreads();
    for (int k = 128; k > 0; k >>= 1) {
        if (threadIdx.x < k) s[threadIdx.x] += s[threadIdx.x + k];
        __syncthreads();
    }
    if (threadIdx.x == 0) f.partial[blockIdx.x] = s[0];
    __syncthreads();
    const double share = gm_share_sum256(f.epart, f.n_epart, s);
    if (threadIdx.x == 0) {
        f.partial[GM_FRAME_BLOCKS + blockIdx.x] = share;
        __threadfence();
        last = atomicAdd(&st->blocks_done, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    const double e_pot = gm_blocks_sum256(f.partial + GM_FRAME_BLOCKS, s);
    if (threadIdx.x == 0) {
        double sum = 0.0;
        for (int b = 0; b < (int)gridDim.x; b++) sum += ((volatile double *)f.partial)[b];
        const double e_kin = 0.5 * sum * (1.0 / (20.455 * 20.455));  // kinetic_final
        st->blocks_done = 0;
        if (store) {
            f.step[slot] = step;
            f.energy[2 * slot] = e_pot;
            f.energy[2 * slot + 1] = e_kin;
            st->frame_n = slot + 1;
        } else {
            st->frame_lost += 1;
        }
    }
}

__global__ void kinetic_final(const double *partial, int blocks, double *out) {
    if (threadIdx.x != 0) return;
    double sum = 0.0;
    for (int b = 0; b < blocks; b++) sum += partial[b];
    *out = 0.5 * sum * (1.0 / (20.455 * 20.455));  // lib.rs:25,76
}

// flag |= 1 when a differs from b anywhere (bit for bit), |= 2 when a holds
// a non-finite value
__global__ void differs_kernel(int n3, const double *a, const double *b, unsigned int *flag) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    int d = 0, bad = 0;
    if (i < n3) {
        d = __double_as_longlong(a[i]) != __double_as_longlong(b[i]);
        bad = !isfinite(a[i]);
    }
    d = __syncthreads_or(d);
    bad = __syncthreads_or(bad);
    if (threadIdx.x == 0 && (d || bad)) atomicOr(flag, (d ? 1u : 0u) | (bad ? 2u : 0u));
}

__global__ void status_reset_kernel(DevStatus *st, int set_step, unsigned long long step, int keep_base) {
    DevStatus z{};
    z.fail_step = ~0ull;
    z.n_rebuilds = st->n_rebuilds;
    z.step = set_step ? step : st->step;
    z.c_steps = st->c_steps;
    z.shake_sum = st->shake_sum;
    z.rattle_sum = st->rattle_sum;
    z.rec_n = st->rec_n;
    z.c_loops = st->c_loops;
    z.frame_n = st->frame_n;
    z.frame_lost = st->frame_lost;
    z.rebuild_base = keep_base ? st->rebuild_base : st->n_rebuilds;
    *st = z;
}

__global__ void forces_out_kernel(int n3, const long long *force, double *out) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n3) out[i] = (double)force[i] * GM_FIX_INV;
}

}  // namespace

// half_kick_kernel, drift_kernel (resync), check_kernel and pack_kernel's
// per-atom work fused for systems without constraints: one atom per thread,
// the same operations in the same order (a rebuild that the check triggers
// packs again with the new grid).  A block that finds a non-finite position marks bad_pending instead of
// error, and the last block moves it to error, so every block of the launch
// reads the error word as it stood before the launch (as the separate kick and
// drift kernels do).
__global__ void kick_drift_check_kernel(int n, double *pos, double *vel, double *dref, long long *force,
                                        const double *inv_mass, double dt_half, double dt, double inv_dt,
                                        const double *ref, double thr_sq, double far_sq, DevStatus *st,
                                        unsigned long long cond, const int *atom_sys, unsigned int *sys_flag,
                                        unsigned int *sys_far, PackArgs pk) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    int need = 0, bad = 0;
    // read by every block before the last block updates them
    const bool err0 = st->error != 0, tail0 = st->tail_pending != 0;
    if (i < n) {
        double np[3];
        if (!err0) {
            const double inv_m = inv_mass[i];
            for (int d = 0; d < 3; d++) {
                const double f = (double)force[d * n + i] * GM_FIX_INV;
                // the previous step's closing half-kick (same forces) when it
                // is pending, then this step's opening one: two additions in
                // the order of the separate kernels
                const double kick = dt_half * f * inv_m * kForceToAccel;
                double v = vel[d * n + i];
                if (tail0) v = v + kick;
                v = v + kick;
                const double p = pos[d * n + i];
                dref[d * n + i] = p;
                np[d] = p + dt * v;
                pos[d * n + i] = np[d];
                vel[d * n + i] = gm_div_by_dt(np[d] - p, dt, inv_dt);
            }
        } else {
            for (int d = 0; d < 3; d++) np[d] = pos[d * n + i];
        }
        // pack_kernel's work for this atom, from the same FP64 position
        const int sl = pk.slot_of[i];
        const GridInfo *g = pk.grid + atom_sys[i];
        gm_pack_record(pk.coord + 2 * sl, np[0] - g->origin[0], np[1] - g->origin[1], np[2] - g->origin[2], pk.qw[i]);
        if (pk.fp64) {
            pk.pos64s[sl] = make_double4(np[0], np[1], np[2], pk.charge64[i]);
            pk.type_sorted[sl] = pk.type[i];
        }
        for (int d = 0; d < 3; d++) force[d * n + i] = 0;
        bad = !(isfinite(np[0]) && isfinite(np[1]) && isfinite(np[2]));
        const double dx = np[0] - ref[i], dy = np[1] - ref[n + i], dz = np[2] - ref[2 * n + i];
        const double d2 = dx * dx + dy * dy + dz * dz;
        need = d2 > thr_sq;
        if (need) sys_flag[atom_sys[i]] = 1u;
        if (gm_moved_far(d2, far_sq)) sys_far[atom_sys[i]] = 1u;
    }
    need = __syncthreads_or(need);
    bad = __syncthreads_or(bad);
    if (threadIdx.x == 0) {
        if (need) atomicOr(&st->rebuild, 1u);
        if (bad) atomicOr(&st->bad_pending, 1u);
        __threadfence();
        const unsigned done = atomicAdd(&st->blocks_done, 1u);
        if (done == gridDim.x - 1) {
            __threadfence();
            const unsigned r = atomicOr(&st->rebuild, 0u);
            st->blocks_done = 0;
            if (atomicExch(&st->bad_pending, 0u)) atomicOr(&st->error, (unsigned)GM_DEV_NONFINITE_POS);
            const unsigned e = atomicOr(&st->error, 0u);
            if (cond) cudaGraphSetConditional((cudaGraphConditionalHandle)cond, (r && !e) ? 1u : 0u);
            // the previous step is complete; this one's closing half-kick is
            // left to the next step's kernel or the finalizer
            if (!err0) {
                if (tail0) st->step += 1;
                st->tail_pending = 1u;
            }
        }
    }
}
// The closing half-kick of the last unconstrained resident step and its step
// count, when pending; the last block clears the flag after every block has
// read it.  With `epart` the first GM_SUM_BLOCKS blocks sum the energy partials
// instead (a launch of its own took 5-7 us of a one-step call).
__global__ void __launch_bounds__(256) kick_tail_kernel(int n, double *vel, const long long *force,
                                                        const double *inv_mass, double dt_half, DevStatus *st,
                                                        const double *epart, int n_epart, double *energy) {
    __shared__ double s[256];
    const int first = epart ? GM_SUM_BLOCKS : 0;
    if ((int)blockIdx.x < first) {
        gm_energy_block(epart, n_epart, energy, s);
        return;
    }
    int i = ((int)blockIdx.x - first) * blockDim.x + threadIdx.x;
    const bool go = st->tail_pending != 0 && st->error == 0;
    if (i < n && go) {
        const double inv_m = inv_mass[i];
        for (int d = 0; d < 3; d++) {
            const double f = (double)force[d * n + i] * GM_FIX_INV;
            vel[d * n + i] += dt_half * f * inv_m * kForceToAccel;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        const unsigned done = atomicAdd(&st->blocks_done, 1u);
        if (done == gridDim.x - first - 1) {
            st->blocks_done = 0;
            if (go) st->step += 1;
            st->tail_pending = 0u;
        }
    }
}
int gm_check_blocks(int n) { return n > 0 ? (n + 255) / 256 : 1; }

void gm_launch_half_kick(int n, double *vel, const long long *force, const double *inv_mass, double dt_half,
                         const DevStatus *st, cudaStream_t s) {
    if (n) half_kick_kernel<<<(n + 255) / 256, 256, 0, s>>>(n, vel, force, inv_mass, dt_half, st);
}

void gm_launch_half_kick_f64(int n, double *vel, const double *force, const double *inv_mass, double dt_half,
                             cudaStream_t s) {
    if (n) half_kick_f64_kernel<<<(n + 255) / 256, 256, 0, s>>>(n, vel, force, inv_mass, dt_half);
}

void gm_launch_drift(int n, double *pos, double *vel, double *dref, double dt, bool resync, const DevStatus *st,
                     cudaStream_t s) {
    if (n) drift_kernel<<<(n + 255) / 256, 256, 0, s>>>(n, pos, vel, dref, dt, resync ? 1 : 0, st);
}

void gm_launch_resync(int n, const double *pos, double *vel, const double *dref, double dt, const DevStatus *st,
                      cudaStream_t s) {
    if (n) resync_kernel<<<(n + 255) / 256, 256, 0, s>>>(n, pos, vel, dref, dt, 1.0 / dt, st);
}

void gm_launch_step(DevStatus *st, cudaStream_t s) { step_kernel<<<1, 1, 0, s>>>(st); }
void gm_launch_kick_drift_check(int n, double *pos, double *vel, double *dref, long long *force,
                                const double *inv_mass, double dt_half, double dt, const double *ref, double thr_sq,
                                double far_sq, DevStatus *st, unsigned long long cond, const int *atom_sys,
                                unsigned int *sys_flag, unsigned int *sys_far, const PackArgs &pk, cudaStream_t s) {
    kick_drift_check_kernel<<<gm_check_blocks(n), 256, 0, s>>>(n, pos, vel, dref, force, inv_mass, dt_half, dt,
                                                              1.0 / dt, ref, thr_sq, far_sq, st, cond, atom_sys,
                                                              sys_flag, sys_far, pk);
}
void gm_launch_kick_tail(int n, double *vel, const long long *force, const double *inv_mass, double dt_half,
                         DevStatus *st, const double *epart, int n_epart, double *energy, cudaStream_t s) {
    kick_tail_kernel<<<gm_check_blocks(n) + (epart ? GM_SUM_BLOCKS : 0), 256, 0, s>>>(n, vel, force, inv_mass, dt_half,
                                                                                     st, epart, n_epart, energy);
}

void gm_launch_check(int n, const double *pos, const double *ref, double thr_sq, double far_sq, DevStatus *st,
                     unsigned long long cond, int blocks, const int *atom_sys, unsigned int *sys_flag,
                     unsigned int *sys_far, cudaStream_t s) {
    check_kernel<<<blocks, 256, 0, s>>>(n, pos, ref, thr_sq, far_sq, st, cond, atom_sys, sys_flag, sys_far);
}

void gm_launch_shake_prepare(const ClusterArgs &c, int n_atoms, const double *dref, cudaStream_t s) {
    if (c.n_clusters == 0) return;
    reset_T<<<1, 1, 0, s>>>(c.status, 0);
    shake_prepare<<<(c.n_constr + 255) / 256, 256, 0, s>>>(c, dref, n_atoms);
}

int gm_launch_shake_solve(const ClusterArgs &c, int n_atoms, double *pos, cudaStream_t s) {
    if (c.n_clusters == 0) return 0;
    // 32-thread blocks over the three cluster ranges: the FP64 pipe of
    // every SM gets a share of the (few) clusters
    const int b = cluster_blocks(c);
    int k = 0;
    if (c.lam0) { warm_start_apply<<<b, 32, 0, s>>>(c, pos, n_atoms); k++; }
    cluster_phase1<false><<<b, 32, 0, s>>>(c, pos, nullptr, n_atoms);
    cluster_phase2<false><<<b, 32, 0, s>>>(c, pos, nullptr, n_atoms);
    return k + 2;
}

void gm_launch_shake(const ClusterArgs &c, int n_atoms, const double *dref, double *pos, cudaStream_t s) {
    gm_launch_shake_prepare(c, n_atoms, dref, s);
    gm_launch_shake_solve(c, n_atoms, pos, s);
}

void gm_launch_rattle(const ClusterArgs &c, int n_atoms, const double *pos, double *vel, bool reset, cudaStream_t s) {
    if (c.n_clusters == 0) return;
    if (reset) reset_T<<<1, 1, 0, s>>>(c.status, 1);
    const int b = cluster_blocks(c);
    cluster_phase1<true><<<b, 32, 0, s>>>(c, const_cast<double *>(pos), vel, n_atoms);
    cluster_phase2<true><<<b, 32, 0, s>>>(c, const_cast<double *>(pos), vel, n_atoms);
}

void gm_solve_step_grid(const ClusterArgs &c, int n_free, int *threads, int *blocks, bool *quads) {
    *blocks = 0;
    int dev = 0, sms = 0, per1 = 0, per2 = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return;
    // four lanes a constraint while every such warp has a scheduler of its own:
    // a step of 1,536 atoms of water (32 warps of lanes) 134 -> 112 us, of 5,184
    // (108) 175 -> 154; of 24,000 (500) it would go from 340 to 379
    const bool comp = c.n_lane_warps <= sms;
    // few constraints: a warp per block, so that every SM's FP64 pipe gets its share
    *threads = c.n_lane_warps <= 4 * sms ? 32 : 128;
    const cudaError_t e1 = comp ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per1, shake_comp_kernel, *threads, 0)
                                : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per1, shake_step_kernel, *threads, 0);
    const cudaError_t e2 = comp ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per2, rattle_comp_kernel, *threads, 0)
                                : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per2, rattle_step_kernel, *threads, 0);
    if (e1 != cudaSuccess || e2 != cudaSuccess) return;
    const int fit = (per1 < per2 ? per1 : per2) * sms, warps = *threads / 32;
    const int need = comp ? 4 * c.n_lane_warps : (c.n_lane_warps + warps - 1) / warps;
    if (need > fit) return;
    *quads = comp;
    // the free atoms take the rest of the SMs, one atom a thread while they last
    const int extra = (n_free + *threads - 1) / *threads;
    *blocks = need + extra < fit ? need + extra : fit;
}

namespace {
template <typename... A>
void launch_cooperative(void (*kernel)(A...), int blocks, int threads, cudaStream_t s, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, args...);
}
}  // namespace

void gm_launch_solve_begin(SolveSync *two, long long todo, cudaStream_t s) {
    solve_begin_kernel<<<1, 1, 0, s>>>(two, todo);
}
void gm_launch_shake_step(const ClusterArgs &c, const SolveStepArgs &sa, const PackArgs &pk, int threads, int blocks,
                          bool quads, cudaStream_t s) {
    launch_cooperative<ClusterArgs, SolveStepArgs, PackArgs>(quads ? shake_comp_kernel : shake_step_kernel, blocks,
                                                             threads, s, c, sa, pk);
}
void gm_launch_rattle_step(const ClusterArgs &c, const SolveStepArgs &sa, int threads, int blocks, bool quads,
                           cudaStream_t s) {
    launch_cooperative<ClusterArgs, SolveStepArgs>(quads ? rattle_comp_kernel : rattle_step_kernel, blocks, threads, s,
                                                   c, sa);
}

void gm_launch_kinetic(int n, const double *vel, const double *mass, double *partials, int blocks, double *out,
                       cudaStream_t s) {
    kinetic_partial<<<blocks, 256, 0, s>>>(n, vel, mass, partials);
    kinetic_final<<<1, 32, 0, s>>>(partials, blocks, out);
}

void gm_launch_frame(int n, const double *pos, const double *vel, const long long *force, const double *inv_mass,
                     const double *mass, double dt_half, DevStatus *st, const FrameArgs &f, cudaStream_t s) {
    frame_kernel<<<GM_FRAME_BLOCKS, 256, 0, s>>>(n, pos, vel, force, inv_mass, mass, dt_half, st, f);
}
void gm_launch_status_reset(DevStatus *st, int set_step, unsigned long long step, int keep_base, cudaStream_t s) {
    status_reset_kernel<<<1, 1, 0, s>>>(st, set_step, step, keep_base);
}
void gm_launch_differs(int n, const double *a, const double *b, unsigned int *flag, cudaStream_t s) {
    if (n) differs_kernel<<<(3 * n + 255) / 256, 256, 0, s>>>(3 * n, a, b, flag);
}

void gm_launch_forces_out(int n, const long long *force, double *out, cudaStream_t s) {
    if (n) forces_out_kernel<<<(3 * n + 255) / 256, 256, 0, s>>>(3 * n, force, out);
}
