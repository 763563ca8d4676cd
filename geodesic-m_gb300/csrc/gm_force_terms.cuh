// gm_force_terms.cuh — the per-item force arithmetic shared by the force
// kernels (gm_force.cu) and the persistent step kernel (gm_step.cu).  Both
// translation units compile these functions with the same flags (FMA
// contraction on), so a force evaluated by either form has the same bits.
//   pair_item_mixed  one warp's share of a 32-atom group's list columns
//   bonded_term      one bond, angle or dihedral (FP64)
//   pair14_term      one scaled 1-4 pair (FP64)
#pragma once
#include "gm_internal.cuh"

namespace {

constexpr int kChunk = 32;
constexpr int kBatch = 4;  // list entries gathered together in the mixed pair kernel

// MUFU approximations of 1/x and 1/sqrt(x); the double-float corrections
// that follow them absorb their few-ulp error.
__device__ __forceinline__ float rcp_approx(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rsqrt_approx(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Minimum image of a pair difference held as dh (a multiple of 2^-8) plus
// dl: the image shift n L is taken with L as a double-float, dh - n L_hi is
// exact (Sterbenz), and the result is put back on the 2^-8 grid so that its
// square stays exact.  n = 0 leaves both unchanged.
__device__ __forceinline__ void image_df(float &dh, float &dl, float L, float Llo, float iL) {
    const float k = rintf(dh * iL);
    dh = fmaf(-k, L, dh);
    dl = fmaf(-k, Llo, dl);
    const float q = rintf(dh * 256.f) * (1.f / 256.f);
    dl += dh - q;
    dh = q;
}

// Difference of two slot records (at the nearest image: `vote` is a warp vote,
// so all lanes call) and its square r^2 as a double-float.
template <bool PERIODIC>
__device__ __forceinline__ gm_df pair_r2(const float4 &mh, const float4 &ml, const float4 &jh, const float4 &jl,
                                         const PairConst &k, float *d_h, float *d_l) {
    d_h[0] = jh.x - mh.x; d_h[1] = jh.y - mh.y; d_h[2] = jh.z - mh.z;
    d_l[0] = jl.x - ml.x; d_l[1] = jl.y - ml.y; d_l[2] = jl.z - ml.z;
    float S = fmaf(d_h[2], d_h[2], fmaf(d_h[1], d_h[1], d_h[0] * d_h[0]));  // exact
    if (PERIODIC) {
        if (__any_sync(0xffffffffu, S > k.img2)) {
#pragma unroll
            for (int d = 0; d < 3; d++) image_df(d_h[d], d_l[d], k.box[d], k.box_lo[d], k.inv_box[d]);
            S = fmaf(d_h[2], d_h[2], fmaf(d_h[1], d_h[1], d_h[0] * d_h[0]));
        }
    }
    const float c = fmaf(d_l[2], fmaf(2.f, d_h[2], d_l[2]),
                         fmaf(d_l[1], fmaf(2.f, d_h[1], d_l[1]), d_l[0] * fmaf(2.f, d_h[0], d_l[0])));
    return gm_fast_sum(S, c);
}

// F_r / r (and with ENERGY the pair energy v) of a pair inside the cutoff:
// R = r^2, p = (sigma^2, 24 epsilon) as double-floats.  Every rounding is
// pinned: the kernels that inline this get the same bits.
template <bool COULOMB, bool ENERGY>
__device__ __forceinline__ void pair_terms(const gm_df R, const gm_df qi, const gm_df qj, const float4 p,
                                           const PairConst &k, gm_df &G, float &v) {
    // 1/r^2 = y (1 + rho - Rl y), rho = 1 - Rh y
    const float y = rcp_approx(R.h);
    const float rho = fmaf(-R.h, y, 1.f);
    const gm_df inv = gm_df_make(y, y * fmaf(-R.l, y, rho));
    // 1/r = z (1 - tau / 2), tau = (Rh + Rl) z^2 - 1 from exact products
    const float z = rsqrt_approx(R.h);
    const float rz = __fmul_rn(R.h, z), ez = fmaf(R.h, z, -rz);
    const float tau = fmaf(R.l, y, fmaf(ez, z, fmaf(rz, z, -1.f)));
    const gm_df rinv = gm_df_make(z, -0.5f * z * tau);
    gm_df Vc = gm_df_make(0.f, 0.f), Gc = Vc;
    if (COULOMB) {
        Vc = gm_dmul(gm_dmul(qi, qj), rinv);  // k q_i q_j / r
        Gc = gm_dmul(Vc, inv);                // (k q_i q_j / r^2) / r
    }
    if (R.h <= k.rsw2) {
        const gm_df x = gm_dmul(gm_df_make(p.x, p.y), inv);  // (sigma / r)^2
        const gm_df x3 = gm_dmul(gm_dsqr(x), x);
        gm_df w2 = gm_two_sum(x3.h + x3.h, -1.f);  // 2 x3 - 1
        w2.l = fmaf(2.f, x3.l, w2.l);
        const gm_df g = gm_dmul(gm_dmul(gm_dmul(gm_df_make(p.z, p.w), x3), w2), inv);
        G = gm_dadd(g, Gc);
        if (ENERGY) v = fmaf(__fmul_rn(__fmul_rn(p.z, 1.f / 6.f), x3.h), x3.h - 1.f, Vc.h + Vc.l);
    } else {
        // LJ in FP32 (tiny here), then V S and F_r S - V dS/dr
        // (products rounded where the compiler could otherwise fuse them
        // into the sums that follow)
        const float xs = p.x * y, x3 = __fmul_rn(__fmul_rn(xs, xs), xs);
        const float vlj = p.z * (1.f / 6.f) * x3 * (x3 - 1.f);
        const float glj = p.z * x3 * fmaf(2.f, x3, -1.f) * y;
        const gm_df V = gm_dadd(Vc, gm_df_make(vlj, 0.f));
        const gm_df G0 = gm_dadd(Gc, gm_df_make(glj, 0.f));
        // r = r^2 / r, whose head and its error are rz and ez
        gm_df u0 = gm_fast_sum(rz, -k.rsw);
        u0.l += fmaf(R.l, z, fmaf(R.h, rinv.l, ez)) - k.rsw_lo;
        const gm_df uu = gm_dmul(u0, gm_df_make(k.inv_w, k.inv_w_lo));
        const gm_df u2 = gm_dsqr(uu), u3 = gm_dmul(u2, uu);
        // S = 1 + u^3 (-10 + u (15 - 6 u))
        const float p6 = __fmul_rn(6.f, uu.h), e6 = fmaf(6.f, uu.h, -p6);
        gm_df t = gm_fast_sum(15.f, -p6);
        t.l -= fmaf(6.f, uu.l, e6);
        t = gm_dmul(uu, t);
        gm_df t3 = gm_fast_sum(-10.f, t.h);
        t3.l += t.l;
        t = gm_dmul(u3, t3);
        gm_df sw = gm_fast_sum(1.f, t.h);
        sw.l += t.l;
        // dS/dr = -30 u^2 (1 - u)^2 / w
        gm_df om = gm_fast_sum(1.f, -uu.h);
        om.l -= uu.l;
        const gm_df ds = gm_dmul(gm_dmul(u2, gm_dsqr(om)), gm_df_make(k.mds, k.mds_lo));
        G = gm_dadd(gm_dmul(G0, sw), gm_dneg(gm_dmul(gm_dmul(V, ds), rinv)));
        if (ENERGY) v = __fmul_rn(V.h + V.l, sw.h + sw.l);
    }
}

// One work item of the mixed-precision nonbonded kernel (force/nonbonded.rs:20-82
// physics plus the switched Coulomb term): FP32 operations throughout, arranged as
// double-float arithmetic so that each pair's force carries ~1e-10 relative
// error (an FP64 pipe is 1/64 of the FP32 one on this part).
//   * Coordinates: each slot holds hi = (x, y, z) rounded to a multiple of
//     2^-8 A and lo = the FP32 remainder.  dh = hj - hi is exact, each dh^2
//     is exact (|dh| < 16 A) and so is their sum S; r^2 = S + c with
//     c = dl (2 dh + dl), renormalised to (Rh, Rl).
//   * Image (periodic): a raw S up to (0.49 box)^2 proves that no component
//     needs one, so a row of 32 pairs pays one comparison and a vote, and the
//     image (24 operations) only where a lane may cross a face.
//   * 1/r^2 and 1/r: MUFU approximations corrected by one residual each.
//   * LJ below the switch radius and the Coulomb term in double-float; the
//     switch polynomial S(u) and dS/du in double-float; LJ inside the switch
//     band (under 1e-2 kcal/mol/A there) in plain FP32.  Sums whose larger
//     term is known take a Fast2Sum (the same two words as the TwoSum, three
//     operations fewer).
//   * F_i -= G d accumulated per lane with TwoSum over chunks of 32 entries;
//     each chunk's (hi, lo) sum is folded into int64 fixed point, so the
//     result is independent of how the columns are split over warps.  (Biased
//     accumulators that take half the operations, and a reassociated switch
//     band, were tried: as exact against FP64, but not the same bits, and a
//     trajectory of rigid-bond water doubles a 1e-10 difference every five
//     steps.)
// Bound: FP32 issue, then the L1 gathers (one wavefront per lane and entry).
// A row of a column takes about 130 instructions inside the switch radius and
// 210 in the band (137 and 231 before, and 24 more of each in a periodic box):
// a step of 98,304 atoms of water executes 397 M warp instructions (479 M).
// The list columns are ordered by build distance (inside the switch radius,
// the switch band, then the shell beyond the cutoff), so a warp's 32 lanes
// usually take the same branch and skip whole regions together.
// Warp w works on group w / split and on the part w % split of the group's
// list columns: entries [part * per, (part + 1) * per), per a multiple of the
// 32-entry chunk.  The split raises the number of warps in flight (a
// 50k-atom system has only 1,563 groups).
// BATCH: systems of a batch have their own type tables ([system][type][type],
// read through L1); a single system keeps its table in shared memory.
// ENERGY false: the item adds its forces only (no energy partial, no
// per-system energy); the force bits are the same.
template <bool PERIODIC, bool COULOMB, bool BATCH, bool ENERGY = true>
__device__ __forceinline__ void
pair_item_mixed(int wid, int lane, int n, int cap, int split, const float4 *__restrict__ coord,
                const int *__restrict__ perm, const int *__restrict__ list, const int *__restrict__ count,
                const int *__restrict__ gmax, const int *__restrict__ count_in, const int *__restrict__ gmax_in,
                const unsigned *__restrict__ sys_far, int ntypes, const float4 *__restrict__ tab, const float4 *s_tab,
                const PairConst &k, long long *__restrict__ force, double *__restrict__ epart, DevStatus *st,
                const int *__restrict__ group_sys, long long *e_sys) {
    const unsigned full = 0xffffffffu;
    const int group = wid / split, part = wid - group * split;
    // without the outer half of the skin while nothing can have come in from it
    const bool inner = sys_far && sys_far[group_sys[group]] == 0u;
    // With energies the parts are those of the whole columns, so that the energy
    // partials hold the same chunks whichever columns a call walks; the forces
    // are the same bits for any parts (98,304 atoms of water, 10 steps: 6,795 us
    // so, 6,845 with the whole columns' parts in every step).
    const int gm = inner ? gmax_in[group] : gmax[group], cols = ENERGY ? gmax[group] : gm;
    const int per = ((cols + split - 1) / split + kChunk - 1) / kChunk * kChunk;
    const int e_begin = part * per, e_end = min(gm, e_begin + per);
    if (e_begin >= e_end) {  // no columns left for this part
        if (ENERGY && lane == 0) epart[wid] = 0.0;
        return;
    }
    const int s = group * 32 + lane;
    const int atom = perm[s];  // -1 on a padding slot
    const bool valid = atom >= 0;
    // a padding lane stands on slot 0 and gathers slot 0: r2 == 0 drops it
    const int self = valid ? s : 0;
    float4 mh, ml;
    gm_ld_coord(coord + 2 * self, mh, ml);
    const int cnt = valid ? (inner ? count_in : count)[s] : 0;
    const float4 *trow = (BATCH ? tab + (size_t)group_sys[group] * ntypes * ntypes : s_tab) +
                         (valid ? gm_slot_type(ml.w) : 0) * ntypes;
    const gm_df qi = gm_df_make(mh.w, ml.w);
    const int *L = list + (size_t)group * 32 * cap + lane;
    long long ax = 0, ay = 0, az = 0;
    double eacc = 0.0;
    unsigned int bad = 0;
    for (int e0 = e_begin; e0 < e_end; e0 += kChunk) {
        gm_df acc[3] = {gm_df_make(0.f, 0.f), gm_df_make(0.f, 0.f), gm_df_make(0.f, 0.f)};
        float ev = 0.f;
        const int e1 = min(e0 + kChunk, e_end);
        for (int e = e0; e < e1; e += kBatch) {
            // lanes past their own count (or the chunk) gather their own
            // atom: r2 == 0 drops it
            int jj[kBatch];
#pragma unroll
            for (int u = 0; u < kBatch; u++)
                jj[u] = (e + u < cnt && e + u < e1) ? __ldg(L + (size_t)(e + u) * 32) : self;
            float4 jhv[kBatch], jlv[kBatch];
#pragma unroll
            for (int u = 0; u < kBatch; u++) gm_ld_coord(coord + 2 * jj[u], jhv[u], jlv[u]);
#pragma unroll
            for (int u = 0; u < kBatch; u++) {
                const float4 jh = jhv[u], jl = jlv[u];
                float d_h[3], d_l[3];
                const gm_df R = pair_r2<PERIODIC>(mh, ml, jh, jl, k, d_h, d_l);
                const bool in = R.h <= k.rc2 && R.h > 0.f;
                if (!__any_sync(full, in)) continue;  // warp-uniform: the shell beyond the cutoff
                if (in) {
                    const float4 p = BATCH ? __ldg(trow + gm_slot_type(jl.w)) : trow[gm_slot_type(jl.w)];
                    gm_df G;  // F_r / r
                    float v;
                    pair_terms<COULOMB, ENERGY>(R, qi, gm_df_make(jh.w, jl.w), p, k, G, v);
                    if (ENERGY) ev += v;
                    // F_i -= G d, each product with its exact error
#pragma unroll
                    for (int d = 0; d < 3; d++) {
                        const float pr = __fmul_rn(G.h, d_h[d]);
                        const float er = fmaf(G.h, d_l[d], fmaf(G.l, d_h[d], fmaf(G.h, d_h[d], -pr)));
                        gm_df sum = gm_two_sum(acc[d].h, -pr);
                        sum.l += acc[d].l - er;
                        acc[d] = sum;
                    }
                }
            }
        }
        ax += gm_to_fix_checked(acc[0].h, bad) + gm_f2fix(acc[0].l);
        ay += gm_to_fix_checked(acc[1].h, bad) + gm_f2fix(acc[1].l);
        az += gm_to_fix_checked(acc[2].h, bad) + gm_f2fix(acc[2].l);
        if (ENERGY) eacc += (double)ev;
    }
    if (valid) {
        gm_atomic_fix_add(force + atom, ax);
        gm_atomic_fix_add(force + n + atom, ay);
        gm_atomic_fix_add(force + 2 * n + atom, az);
    }
    if (ENERGY) {
        for (int o = 16; o > 0; o >>= 1) eacc += __shfl_xor_sync(full, eacc, o);
        if (lane == 0) epart[wid] = 0.5 * eacc;
        if (e_sys && lane == 0)
            gm_atomic_fix_add(e_sys + group_sys[group], __double2ll_rn(0.5 * eacc * GM_EFIX_SCALE));
    }
    bad = __reduce_or_sync(full, bad);
    if (bad && lane == 0) atomicOr(&st->error, bad);
}

// Transposes x over the 4 lanes of a quad: lane c of the quad gets x[c] of its
// lanes 0..3, in order.
__device__ __forceinline__ void quad_transpose(float x[4], int sub) {
    const unsigned full = 0xffffffffu;
    const bool b0 = sub & 1, b1 = sub & 2;
    const float p = __shfl_xor_sync(full, b0 ? x[0] : x[1], 1), q = __shfl_xor_sync(full, b0 ? x[2] : x[3], 1);
    if (b0) { x[0] = p; x[2] = q; }
    else { x[1] = p; x[3] = q; }
    const float r = __shfl_xor_sync(full, b1 ? x[0] : x[2], 2), t = __shfl_xor_sync(full, b1 ? x[1] : x[3], 2);
    if (b1) { x[0] = r; x[1] = t; }
    else { x[2] = r; x[3] = t; }
}

// The same work item by a block of four warps, for systems whose items do not
// fill the chip: an item is then one warp's latency, 32 entries of ~1,300
// cycles each (a dependent chain of ~200 FP32 operations).  Here a warp takes 8
// of the group's atoms and four lanes an atom: the four evaluate four
// consecutive entries at once, and after a transposition lane 0, 1, 2 of the
// quad add the four products to the x, y, z sum one after the other (lane 3 the
// energies), in the order and the arithmetic of pair_item_mixed, so every
// sum has its bits.  All threads of the block call; `s_e`: 32 doubles.
template <bool PERIODIC, bool COULOMB, bool ENERGY>
__device__ __forceinline__ void
pair_item_quad(int wid, int warp, int lane, const ForceArgs &fa, const float4 *s_tab, double *s_e) {
    const unsigned full = 0xffffffffu;
    const PairConst &k = fa.pc;
    const int split = fa.split, group = wid / split, part = wid - group * split;
    const bool inner = fa.sys_far && fa.sys_far[fa.group_sys[group]] == 0u;
    const int gm = inner ? fa.gmax_in[group] : fa.gmax[group], cols = ENERGY ? fa.gmax[group] : gm;
    const int per = ((cols + split - 1) / split + kChunk - 1) / kChunk * kChunk;
    const int e_begin = part * per, e_end = min(gm, e_begin + per);
    if (e_begin >= e_end) {  // block-uniform: no columns left for this part
        if (ENERGY && warp == 0 && lane == 0) fa.epart[wid] = 0.0;
        return;
    }
    const int sub = lane & 3, l = warp * 8 + (lane >> 2);
    const int s = group * 32 + l;
    const int atom = fa.perm[s];
    const bool valid = atom >= 0;
    const int self = valid ? s : 0;
    float4 mh, ml;
    gm_ld_coord_rw(fa.coord + 2 * self, mh, ml);
    const int cnt = valid ? (inner ? fa.count_in : fa.count)[s] : 0;
    const float4 *trow = s_tab + (valid ? gm_slot_type(ml.w) : 0) * fa.ntypes;
    const gm_df qi = gm_df_make(mh.w, ml.w);
    const int *L = fa.list + (size_t)group * 32 * fa.cap + l;
    long long sum = 0;
    double eacc = 0.0;
    unsigned bad = 0;
    for (int e0 = e_begin; e0 < e_end; e0 += kChunk) {
        gm_df acc = gm_df_make(0.f, 0.f);
        float ev = 0.f;
        const int e1 = min(e0 + kChunk, e_end);
        int jj[kChunk / 4];
#pragma unroll
        for (int t = 0; t < kChunk / 4; t++) {
            const int e = e0 + 4 * t + sub;
            jj[t] = e < cnt && e < e1 ? __ldg(L + (size_t)e * 32) : self;
        }
        float4 jh, jl, nh, nl;
        gm_ld_coord_rw(fa.coord + 2 * jj[0], nh, nl);
#pragma unroll
        for (int t = 0; t < kChunk / 4; t++) {
            jh = nh;
            jl = nl;
            if (t + 1 < kChunk / 4) gm_ld_coord_rw(fa.coord + 2 * jj[t + 1], nh, nl);  // beside these entries' arithmetic
            float d_h[3], d_l[3];
            const gm_df R = pair_r2<PERIODIC>(mh, ml, jh, jl, k, d_h, d_l);
            const bool in = R.h <= k.rc2 && R.h > 0.f;
            if (!__any_sync(full, in)) continue;
            // an entry outside adds zeros, which change no sum
            float pr[4] = {0.f, 0.f, 0.f, 0.f}, er[4] = {0.f, 0.f, 0.f, 0.f};
            if (in) {
                gm_df G;
                float v = 0.f;
                pair_terms<COULOMB, ENERGY>(R, qi, gm_df_make(jh.w, jl.w), trow[gm_slot_type(jl.w)], k, G, v);
#pragma unroll
                for (int d = 0; d < 3; d++) {
                    pr[d] = __fmul_rn(G.h, d_h[d]);
                    er[d] = fmaf(G.h, d_l[d], fmaf(G.l, d_h[d], fmaf(G.h, d_h[d], -pr[d])));
                }
                if (ENERGY) pr[3] = v;
            }
            quad_transpose(pr, sub);
            quad_transpose(er, sub);
#pragma unroll
            for (int q = 0; q < 4; q++) {
                gm_df t2 = gm_two_sum(acc.h, -pr[q]);
                t2.l += acc.l - er[q];
                acc = t2;
                if (ENERGY) ev += pr[q];
            }
        }
        if (sub < 3) sum += gm_to_fix_checked(acc.h, bad) + gm_f2fix(acc.l);
        else if (ENERGY) eacc += (double)ev;
    }
    if (valid && sub < 3) gm_atomic_fix_add(fa.force + (size_t)sub * fa.n + atom, sum);
    if (ENERGY) {
        __syncthreads();
        if (sub == 3) s_e[l] = eacc;
        __syncthreads();
        if (warp == 0) {
            double e = s_e[lane];
            for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(full, e, o);
            if (lane == 0) fa.epart[wid] = 0.5 * e;
        }
    }
    bad = __reduce_or_sync(full, bad);
    if (bad && lane == 0) atomicOr(&fa.status->error, bad);
}

// ----------------------------------------------------------------- bonded
//
// Bond, angle and dihedral terms and the scaled 1-4 pairs run in FP64 in both
// precisions: they are ~3N terms against ~400N pair evaluations, and their
// forces (k = 300 bonds balancing the LJ repulsion of a dense lattice) are
// large enough that FP32 rounding alone would exceed 1e-5 of a small net
// force.

struct V3 { double x, y, z; };

// pos[ia] - pos[ib] in FP64; with MI at the nearest periodic image (the
// reference's min_image on each component)
template <bool MI>
__device__ __forceinline__ V3 pdiff(const ForceArgs &a, int ia, int ib) {
    const int n = a.n;
    V3 d = {a.pos[ia] - a.pos[ib], a.pos[n + ia] - a.pos[n + ib], a.pos[2 * n + ia] - a.pos[2 * n + ib]};
    if constexpr (MI) {
        d.x = gm_min_image(d.x, a.box64[0]);
        d.y = gm_min_image(d.y, a.box64[1]);
        d.z = gm_min_image(d.z, a.box64[2]);
    }
    return d;
}
// The FP64 term arithmetic below fixes every fused multiply-add itself
// (fma where a product feeds a sum, __dmul_rn where a product must stay
// rounded): the compiler's own contraction choices may differ between the
// kernels that inline these functions, and both step forms must round alike.
__device__ __forceinline__ double pmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ V3 cross(V3 a, V3 b) {
    return {fma(a.y, b.z, -pmul(a.z, b.y)), fma(a.z, b.x, -pmul(a.x, b.z)), fma(a.x, b.y, -pmul(a.y, b.x))};
}
__device__ __forceinline__ double dot(V3 a, V3 b) { return fma(a.z, b.z, fma(a.y, b.y, pmul(a.x, b.x))); }

__device__ __forceinline__ void add_force(long long *f, int n, int a, double x, double y, double z, unsigned &bad) {
    gm_atomic_fix_add(f + a, gm_to_fix_checked(x, bad));
    gm_atomic_fix_add(f + n + a, gm_to_fix_checked(y, bad));
    gm_atomic_fix_add(f + 2 * n + a, gm_to_fix_checked(z, bad));
}

// Term t of the bonded list (bonds, then angles, then dihedrals; t past the
// end is no term): adds its forces and returns its energy; `first` is an atom
// of the term (its system owns the energy).
template <bool MI>
__device__ __forceinline__ double bonded_term(const ForceArgs &a, int t, unsigned &bad, int &first) {
    const int n = a.n;
    double e = 0.0;
    if (t < a.n_bonds) {
        // force/bonded.rs:5-40, V = k (r - r0)^2
        const int i = a.bond_i[t], j = a.bond_j[t];
        first = i;
        const V3 d = pdiff<MI>(a, j, i);
        const double k = a.bond_k[t], r0 = a.bond_r0[t];
        const double r2 = dot(d, d);
        if (r2 > 0.0) {
            const double ir = rsqrt(r2);
            const double dr = fma(r2, ir, -r0);
            e = pmul(pmul(k, dr), dr);
            const double g = pmul(pmul(pmul(2.0, k), dr), ir);
            const double gx = pmul(g, d.x), gy = pmul(g, d.y), gz = pmul(g, d.z);
            add_force(a.force, n, i, gx, gy, gz, bad);
            add_force(a.force, n, j, -gx, -gy, -gz, bad);
        }
    } else if (t < a.n_bonds + a.n_angles) {
        // force/bonded.rs:44-102, V = k (theta - theta0)^2
        const int q = t - a.n_bonds;
        const int i = a.angle_i[q], j = a.angle_j[q], kk = a.angle_k[q];
        first = i;
        const V3 b1 = pdiff<MI>(a, i, j), b2 = pdiff<MI>(a, kk, j);
        const double q1 = dot(b1, b1), q2 = dot(b2, b2);
        if (q1 != 0.0 && q2 != 0.0) {
            const double i1 = rsqrt(q1), i2 = rsqrt(q2);
            double c = pmul(pmul(dot(b1, b2), i1), i2);
            c = c < -1.0 ? -1.0 : (c > 1.0 ? 1.0 : c);
            double sn = sqrt(fma(-c, c, 1.0));
            sn = sn > 1e-8 ? sn : 1e-8;
            const double dth = acos(c) - a.angle_th0[q];
            const double k = a.angle_kth[q];
            e = pmul(pmul(k, dth), dth);
            const double aa = pmul(pmul(2.0, k), dth) / sn;
            const double ir12 = pmul(i1, i2), ir11 = pmul(i1, i1), ir22 = pmul(i2, i2);
            // aa (b2 / (|b1| |b2|) - c b1 / |b1|^2), and the same for k
            const V3 fi = {pmul(aa, fma(b2.x, ir12, -pmul(pmul(c, b1.x), ir11))),
                           pmul(aa, fma(b2.y, ir12, -pmul(pmul(c, b1.y), ir11))),
                           pmul(aa, fma(b2.z, ir12, -pmul(pmul(c, b1.z), ir11)))};
            const V3 fk = {pmul(aa, fma(b1.x, ir12, -pmul(pmul(c, b2.x), ir22))),
                           pmul(aa, fma(b1.y, ir12, -pmul(pmul(c, b2.y), ir22))),
                           pmul(aa, fma(b1.z, ir12, -pmul(pmul(c, b2.z), ir22)))};
            add_force(a.force, n, i, fi.x, fi.y, fi.z, bad);
            add_force(a.force, n, kk, fk.x, fk.y, fk.z, bad);
            add_force(a.force, n, j, -(fi.x + fk.x), -(fi.y + fk.y), -(fi.z + fk.z), bad);
        }
    } else if (t < a.n_bonds + a.n_angles + a.n_diheds) {
        // force/bonded.rs:112-164, V = k [1 + cos(n phi - delta)]
        const int q = t - a.n_bonds - a.n_angles;
        const int i = a.dihed_i[q], j = a.dihed_j[q], k = a.dihed_k[q], l = a.dihed_l[q];
        first = i;
        const V3 b1 = pdiff<MI>(a, j, i), b2 = pdiff<MI>(a, k, j), b3 = pdiff<MI>(a, l, k);
        const V3 m = cross(b1, b2), nv = cross(b2, b3);
        const double m2 = dot(m, m), n2 = dot(nv, nv), b22 = dot(b2, b2);
        if (m2 != 0.0 && n2 != 0.0 && b22 != 0.0) {
            const double ib2 = rsqrt(b22), b2l = pmul(b22, ib2);
            // phi = atan2(y, x) as in the reference; cos(n phi - delta) and
            // sin(n phi - delta) are taken without the transcendentals:
            // (cos phi, sin phi) = (x, y) / |(x, y)|, raised to the n-th
            // power as a complex number, then rotated by delta (the FP64
            // pipe of this part is 1/64 of its FP32 one)
            const double x = dot(m, nv);
            const double y = pmul(dot(cross(m, nv), b2), ib2);
            const double ir = rsqrt(fma(x, x, pmul(y, y)));
            const double c1 = pmul(x, ir), s1 = pmul(y, ir);
            const unsigned mult = a.dihed_n[q];
            double cn = 1.0, sn = 0.0;
            for (unsigned it = 0; it < mult; it++) {
                const double c2 = fma(cn, c1, -pmul(sn, s1));
                sn = fma(sn, c1, pmul(cn, s1));
                cn = c2;
            }
            const double2 cs = a.dihed_cs[q];  // (cos delta, sin delta)
            const double kphi = a.dihed_kphi[q];
            e = pmul(kphi, 1.0 + fma(cn, cs.x, pmul(sn, cs.y)));
            const double dv = pmul(pmul(kphi, (double)mult), fma(sn, cs.x, -pmul(cn, cs.y)));  // -dV/dphi
            const double imn = pmul(dv, b2l) / pmul(m2, n2);
            const double si = pmul(-imn, n2), sl = pmul(imn, m2);
            const V3 fi = {pmul(m.x, si), pmul(m.y, si), pmul(m.z, si)};
            const V3 fl = {pmul(nv.x, sl), pmul(nv.y, sl), pmul(nv.z, sl)};
            const double ib = pmul(ib2, ib2);
            const double p = pmul(dot(b1, b2), ib), qq = pmul(dot(b3, b2), ib);
            const double p1 = -(p + 1.0), q1 = qq + 1.0;
            const V3 fj = {fma(qq, fl.x, pmul(p1, fi.x)), fma(qq, fl.y, pmul(p1, fi.y)), fma(qq, fl.z, pmul(p1, fi.z))};
            const V3 fk = {fma(p, fi.x, -pmul(q1, fl.x)), fma(p, fi.y, -pmul(q1, fl.y)), fma(p, fi.z, -pmul(q1, fl.z))};
            add_force(a.force, n, i, fi.x, fi.y, fi.z, bad);
            add_force(a.force, n, j, fj.x, fj.y, fj.z, bad);
            add_force(a.force, n, k, fk.x, fk.y, fk.z, bad);
            add_force(a.force, n, l, fl.x, fl.y, fl.z, bad);
        }
    }
    return e;
}

// Scaled 1-4 pair t (beyond the reference): unswitched, no cutoff; LJ scaled
// by scale14_lj, Coulomb by scale14_coul.
template <bool MI>
__device__ __forceinline__ double pair14_term(const ForceArgs &a, int t, unsigned &bad, int &first) {
    const int n = a.n;
    double e = 0.0;
    if (t < a.n14) {
        const int i = a.p14_i[t], j = a.p14_j[t];
        first = i;
        const V3 d = pdiff<MI>(a, j, i);
        const double r2 = dot(d, d);
        if (r2 > 0.0) {
            // (sigma_ij, 4 eps_ij s_lj, 24 eps_ij s_lj, k_C q_i q_j s_coul)
            const double4 p = a.p14par[t];
            const double rinv = rsqrt(r2);
            const double sr = pmul(p.x, rinv), s2 = pmul(sr, sr), s4 = pmul(s2, s2), s6 = pmul(s2, s4);
            const double s12 = pmul(s6, s6);
            const double vc = pmul(p.w, rinv);
            e = fma(p.y, s12 - s6, vc);
            const double g = pmul(pmul(fma(p.z, fma(2.0, s12, -s6), vc), rinv), rinv);
            const double gx = pmul(g, d.x), gy = pmul(g, d.y), gz = pmul(g, d.z);
            add_force(a.force, n, i, -gx, -gy, -gz, bad);
            add_force(a.force, n, j, gx, gy, gz, bad);
        }
    }
    return e;
}

}  // namespace
