// gm_step.cu — the unconstrained mixed-precision BAB step (lib.rs:292-323
// without constraints) as one persistent cooperative launch per step.
//
// Launch k of a run starts from the positions x_k that launch k-1 left (and
// the list that the graph's conditional rebuild left after it):
//   1. forces F(x_k): every warp takes work items from one queue: the pair
//      items of the mixed kernel (pair_item_mixed, a 32-atom group's share of
//      list columns) and chunks of the bonded terms and 1-4 pairs (128 terms,
//      32 in a small system),
//      spread evenly through the queue so that each SM mixes FP32 pair work
//      with FP64 bonded work.  Skipped when the forces at x_k are summed
//      already (the first launch of a call: the call starts with current
//      forces).
//   2. one grid barrier (bounded: a block that waits too long records
//      GM_DEV_BARRIER_TIMEOUT and returns).
//   3. per atom, grid-strided: the closing half-kick of step k-1 (when
//      pending) and the opening half-kick of step k with F(x_k), the drift to
//      x_{k+1}, the velocity resync, the pack of x_{k+1}, the zeroing of the
//      force sums and the rebuild check; the last block sets the graph's
//      rebuild condition.
// The graph that holds the launch has one more node, the IF node of the list
// rebuild.
//
// A small system (QUAD: up to 100 groups) gives a pair item to a block, takes a
// component per lane in phase 3, and runs up to GM_LOOP_STEPS steps a launch: a
// second grid barrier ends each step, and its last block decides whether the
// launch goes on (no rebuild, no error, steps left).  The call is one graph:
// WHILE steps are left, the launch, IF rebuild.  50 steps of 224 atoms: 1,902 us
// with a launch a step, 1,471 so, 1,420 with phase 3 a component per lane.
// Larger systems keep a launch a step: coordinates that the launch itself writes
// cannot be read through the read-only path, and without it 98,304 atoms were
// 1.5 % and 786,432 1.6 % slower.
//
// After the last launch of a call the forces F(x_n) are evaluated
// by this kernel's force phase alone (the STEP = false instantiation, with
// energies) and the closing half-kick by the tail kernel, so a call ends as
// in the kernel-graph form.
//
// The launch performs the kernel-graph form's operations in the same order:
// force sums are integer sums (the order of the work items changes no bit),
// and phase 3 is written with explicit round-to-nearest operations, so it
// rounds like the integrator kernels, which are compiled without
// contraction.  Energies are not evaluated inside the loop (the force
// evaluation after the last launch sums them): the pair items and the
// bonded chunks add forces only.
#include "gm_force_terms.cuh"

namespace {

constexpr int kStepThreads = 128;
constexpr int kStepMinBlocks = 6;  // 24 warps per SM: at most 80 registers a thread
// A 64-term block of bonded terms (or 1-4 pairs) by one warp, two terms a
// lane, with the energy partial and the per-system energies of term_block
// (gm_force.cu): lane l holds terms l and l + 32, and the shuffle-down tree
// adds in the order of its shared-memory tree, so the partial has the same
// bits.
template <bool MI, bool P14>
__device__ __forceinline__ void term_block_warp(const ForceArgs &fa, int blk, int lane, unsigned &bad) {
    int f0 = -1, f1 = -1;
    const int t = blk * GM_BONDED_THREADS + lane;
    const double e0 = P14 ? pair14_term<MI>(fa, t, bad, f0) : bonded_term<MI>(fa, t, bad, f0);
    const double e1 = P14 ? pair14_term<MI>(fa, t + 32, bad, f1) : bonded_term<MI>(fa, t + 32, bad, f1);
    if (fa.e_sys) {
        gm_add_sys_energy(fa.e_sys, f0 >= 0 ? fa.atom_sys[f0] : -1, e0);
        gm_add_sys_energy(fa.e_sys, f1 >= 0 ? fa.atom_sys[f1] : -1, e1);
    }
    double v = e0 + e1;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0 && blk < (P14 ? fa.blocks14 : fa.bonded_blocks)) (P14 ? fa.epart14 : fa.epart_bonded)[blk] = v;
}

// Terms of a bonded ticket: the force phase alone keeps whole 64-term blocks
// (their energy partials).
template <bool STEP>
__host__ __device__ __forceinline__ int ticket_terms(const ForceArgs &fa) {
    return !STEP && fa.term_chunk < GM_BONDED_THREADS ? GM_BONDED_THREADS : fa.term_chunk;
}
__host__ __device__ __forceinline__ int bonded_tickets(const ForceArgs &fa, int chunk) {
    return (fa.n_bonds + fa.n_angles + fa.n_diheds + chunk - 1) / chunk;
}
__host__ __device__ __forceinline__ int pair14_tickets(const ForceArgs &fa, int chunk) {
    return (fa.n14 + chunk - 1) / chunk;
}

// The force phase of a small system (QUAD): a block per pair item
// (pair_item_quad) or per 128 bonded terms, handed out by block index.  With a
// warp per item and a queue the phase was the longest item: 45,000 cycles at
// 1,536 atoms, while most of the chip was idle (34.8 us, now 27.0).
template <bool PERIODIC, bool COULOMB, bool MI, bool STEP>
__device__ __forceinline__ void quad_phase(const ForceArgs &fa, const float4 *s_tab) {
    __shared__ double s_e[kStepThreads];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int cb = bonded_tickets(fa, kStepThreads), nbw = cb + pair14_tickets(fa, kStepThreads);
    const int total = nbw + fa.n_groups * fa.split;
    for (int t = blockIdx.x; t < total; t += gridDim.x) {
        if (t >= nbw) {
            pair_item_quad<PERIODIC, COULOMB, !STEP>(t - nbw, warp, lane, fa, s_tab, s_e);
            continue;
        }
        unsigned bad = 0;
        int first = -1;
        const bool b14 = t >= cb;
        const int term = (b14 ? t - cb : t) * kStepThreads + (int)threadIdx.x;
        const double e = b14 ? pair14_term<MI>(fa, term, bad, first) : bonded_term<MI>(fa, term, bad, first);
        if (!STEP) {
            // term_block's partial of each 64 terms: two warps hold its halves
            __syncthreads();
            s_e[threadIdx.x] = e;
            __syncthreads();
            double v = e + s_e[(threadIdx.x + 32) % kStepThreads];
            for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
            const int blk = term / GM_BONDED_THREADS;
            if (lane == 0 && (warp & 1) == 0 && blk < (b14 ? fa.blocks14 : fa.bonded_blocks))
                (b14 ? fa.epart14 : fa.epart_bonded)[blk] = v;
        }
        bad = __reduce_or_sync(0xffffffffu, bad);
        if (bad && lane == 0) atomicOr(&fa.status->error, bad);
    }
}

// STEP: one BAB step (phases 1-3 above, a cooperative launch).  !STEP: phase
// 1 alone with energies (the pair items' partials, the 64-term blocks'
// partials and the per-system energies of the force kernels, the same bits),
// a plain launch; its last warp clears the queue words.
template <bool PERIODIC, bool COULOMB, bool BATCH, bool MI, bool STEP, bool QUAD>
__global__ void __launch_bounds__(kStepThreads, kStepMinBlocks)
step_persistent_kernel(ForceArgs fa, StepArgs sa, PackArgs pk) {
    extern __shared__ float4 s_tab[];
    DevStatus *st = fa.status;
    StepSync *sy = sa.sync;
    const int lane = threadIdx.x & 31;
    const unsigned full = 0xffffffffu;
    // read by every block before the first barrier; block 0 clears it after
    const bool fresh = STEP && sy->fresh != 0;
    const bool loop = STEP && QUAD && sa.loop;
    const long long todo = loop ? sy->todo : 1;
    const int steps = (int)(todo < GM_LOOP_STEPS ? todo : GM_LOOP_STEPS);
    if (loop && blockIdx.x == 0 && threadIdx.x == 0) {
        // until the last step's bookkeeping says otherwise (a barrier that
        // times out ends the WHILE node)
        cudaGraphSetConditional((cudaGraphConditionalHandle)sa.loop, 0u);
        cudaGraphSetConditional((cudaGraphConditionalHandle)sa.cond, 0u);
    }
    if (!BATCH && !(fresh && steps == 1)) {
        for (int t = threadIdx.x; t < fa.ntypes * fa.ntypes; t += blockDim.x) s_tab[t] = fa.tab32[t];
        __syncthreads();
    }
    for (int k = 0; k < steps; k++) {
        // ---- 1. forces at the current positions
        if (!fresh || k > 0) {
            if constexpr (QUAD) {
                quad_phase<PERIODIC, COULOMB, MI, STEP>(fa, s_tab);
            } else {
            // tickets: n_pair pair items and nbw bonded tickets (chunk bonded
            // terms or 1-4 pairs each), the bonded ones at t = k * stride
            const int n_pair = fa.n_groups * fa.split;
            const int chunk = ticket_terms<STEP>(fa), cb = bonded_tickets(fa, chunk);
            const int nbw = cb + pair14_tickets(fa, chunk), total = n_pair + nbw;
            const int stride = nbw > 0 ? total / nbw : 1;
            for (;;) {
                int t = 0;
                if (lane == 0) t = (int)atomicAdd(&sy->ticket, 1u);
                t = __shfl_sync(full, t, 0);
                if (t >= total) break;
                const int q = t / stride, r = t - q * stride;
                if (r == 0 && q < nbw) {
                    unsigned bad = 0;
                    const bool b14 = q >= cb;
                    if (STEP) {
                        int first = -1;
                        const int base = (b14 ? q - cb : q) * chunk + lane;
                        for (int u = 0; u < chunk; u += 32) {
                            if (b14) pair14_term<MI>(fa, base + u, bad, first);
                            else bonded_term<MI>(fa, base + u, bad, first);
                        }
                    } else {
                        const int blk0 = (b14 ? q - cb : q) * (chunk / GM_BONDED_THREADS);
                        for (int h = 0; h < chunk / GM_BONDED_THREADS; h++) {
                            if (b14) term_block_warp<MI, true>(fa, blk0 + h, lane, bad);
                            else term_block_warp<MI, false>(fa, blk0 + h, lane, bad);
                        }
                    }
                    bad = __reduce_or_sync(full, bad);
                    if (bad && lane == 0) atomicOr(&st->error, bad);
                } else {
                    // bonded tickets at or before t: min(q + 1, nbw)
                    const int item = t - min(q + 1, nbw);
                    pair_item_mixed<PERIODIC, COULOMB, BATCH, !STEP>(
                        item, lane, fa.n, fa.cap, fa.split, fa.coord, fa.perm, fa.list, fa.count, fa.gmax, fa.count_in,
                        fa.gmax_in, fa.sys_far, fa.ntypes, fa.tab32, s_tab, fa.pc, fa.force, fa.epart, st, fa.group_sys,
                        STEP ? nullptr : fa.e_sys);
                }
            }
            }
        }
        if (!STEP) {
            if (QUAD) return;  // no queue
            // the last warp out leaves the queue words at zero for the next launch
            if (lane == 0) {
                __threadfence();
                const unsigned warps = gridDim.x * (blockDim.x / 32);
                if (atomicAdd(&sy->arrive, 1u) == warps - 1) {
                    atomicExch(&sy->ticket, 0u);
                    atomicExch(&sy->arrive, 0u);
                }
            }
            return;
        }
        // ---- 2. every force is summed
        if (!gm_grid_barrier(&sy->arrive, &sy->gen, st)) return;
        // ---- 3. kick, drift, pack, rebuild check (kick_drift_check_kernel's
        // operations, one atom at a time)
        const bool err0 = gm_ld_acquire(&st->error) != 0, tail0 = gm_ld_acquire(&st->tail_pending) != 0;
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            sy->ticket = 0;
            sy->fresh = 0;
        }
        const int n = sa.n;
        int need = 0, bad = 0;
        if constexpr (QUAD) {
            // a component per lane, the fourth lane the charge: an FP64
            // instruction costs a scheduler the same for one lane as for 32,
            // and a small system has schedulers to spare
            for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < ((4 * n + 31) & ~31); e += gridDim.x * blockDim.x) {
                const int i = e >> 2, d = e & 3;
                int sys = 0;
                double dx = 0.0;
                if (i < n) {
                    sys = sa.atom_sys[i];
                    float *rec = reinterpret_cast<float *>(pk.coord + 2 * pk.slot_of[i]);
                    if (d < 3) {
                        const double p = sa.pos[d * n + i];
                        double np = p;
                        if (!err0) {
                            const double f = __dmul_rn((double)__ldcg(fa.force + d * n + i), GM_FIX_INV);
                            const double kick =
                                __dmul_rn(__dmul_rn(__dmul_rn(sa.dt_half, f), sa.inv_mass[i]), GM_FORCE_TO_ACCEL);
                            double v = sa.vel[d * n + i];
                            if (tail0) v = __dadd_rn(v, kick);
                            v = __dadd_rn(v, kick);
                            sa.dref[d * n + i] = p;
                            np = __dadd_rn(p, __dmul_rn(sa.dt, v));
                            sa.pos[d * n + i] = np;
                            sa.vel[d * n + i] = gm_div_by_dt(__dsub_rn(np, p), sa.dt, sa.inv_dt);
                        }
                        gm_pack_component(rec + d, __dsub_rn(np, pk.grid[sys].origin[d]));
                        fa.force[d * n + i] = 0;
                        bad |= !isfinite(np);
                        dx = __dsub_rn(np, sa.ref[d * n + i]);
                    } else {
                        const float2 qw = pk.qw[i];
                        rec[3] = qw.x;
                        rec[7] = qw.y;
                    }
                }
                const double sq = __dmul_rn(dx, dx);
                const double d2 = __dadd_rn(__dadd_rn(__shfl_sync(full, sq, 0, 4), __shfl_sync(full, sq, 1, 4)),
                                            __shfl_sync(full, sq, 2, 4));
                if (i < n) {
                    if (gm_moved_far(d2, sa.far_sq)) sa.sys_far[sys] = 1u;
                    if (d2 > sa.thr_sq) {
                        sa.sys_flag[sys] = 1u;
                        need = 1;
                    }
                }
            }
        } else {
            for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
                double np[3];
                if (!err0) {
                    const double inv_m = sa.inv_mass[i];
                    for (int d = 0; d < 3; d++) {
                        const double f = __dmul_rn((double)__ldcg(fa.force + d * n + i), GM_FIX_INV);
                        const double kick = __dmul_rn(__dmul_rn(__dmul_rn(sa.dt_half, f), inv_m), GM_FORCE_TO_ACCEL);
                        double v = sa.vel[d * n + i];
                        if (tail0) v = __dadd_rn(v, kick);
                        v = __dadd_rn(v, kick);
                        const double p = sa.pos[d * n + i];
                        sa.dref[d * n + i] = p;
                        np[d] = __dadd_rn(p, __dmul_rn(sa.dt, v));
                        sa.pos[d * n + i] = np[d];
                        sa.vel[d * n + i] = gm_div_by_dt(__dsub_rn(np[d], p), sa.dt, sa.inv_dt);
                    }
                } else {
                    for (int d = 0; d < 3; d++) np[d] = sa.pos[d * n + i];
                }
                const int sl = pk.slot_of[i];
                const GridInfo *g = pk.grid + sa.atom_sys[i];
                gm_pack_record(pk.coord + 2 * sl, __dsub_rn(np[0], g->origin[0]), __dsub_rn(np[1], g->origin[1]),
                               __dsub_rn(np[2], g->origin[2]), pk.qw[i]);
                for (int d = 0; d < 3; d++) fa.force[d * n + i] = 0;
                bad |= !(isfinite(np[0]) && isfinite(np[1]) && isfinite(np[2]));
                const double dx = __dsub_rn(np[0], sa.ref[i]), dy = __dsub_rn(np[1], sa.ref[n + i]),
                             dz = __dsub_rn(np[2], sa.ref[2 * n + i]);
                const double d2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
                const bool moved = d2 > sa.thr_sq;
                if (gm_moved_far(d2, sa.far_sq)) sa.sys_far[sa.atom_sys[i]] = 1u;
                if (moved) {
                    sa.sys_flag[sa.atom_sys[i]] = 1u;
                    need = 1;
                }
            }
        }
        need = __syncthreads_or(need);
        bad = __syncthreads_or(bad);
        // ---- 4. the last block's bookkeeping; with steps left, a second barrier
        // whose last block decides for all whether to go on (no block reads the
        // error or rebuild words themselves, which a faster block may set already)
        const bool last_step = !QUAD || k + 1 == steps;
        __shared__ int s_more;
        if (threadIdx.x == 0) {
            if (need) atomicOr(&st->rebuild, 1u);
            if (bad) atomicOr(&st->bad_pending, 1u);
            const unsigned gen = QUAD ? gm_ld_acquire(&sy->gen) : 0u;
            __threadfence();
            const unsigned done = atomicAdd(&st->blocks_done, 1u);
            if (done == gridDim.x - 1) {
                __threadfence();
                const unsigned r = atomicOr(&st->rebuild, 0u);
                st->blocks_done = 0;
                if (atomicExch(&st->bad_pending, 0u)) atomicOr(&st->error, (unsigned)GM_DEV_NONFINITE_POS);
                const unsigned e = atomicOr(&st->error, 0u);
                const bool more = !last_step && !r && !e;
                if (!more) {
                    if (sa.cond) cudaGraphSetConditional((cudaGraphConditionalHandle)sa.cond, (r && !e) ? 1u : 0u);
                    if (loop) {
                        const long long left = todo - (k + 1);
                        sy->todo = left;
                        st->c_loops += 1;
                        cudaGraphSetConditional((cudaGraphConditionalHandle)sa.loop, (left > 0 && !e) ? 1u : 0u);
                    }
                }
                if (!err0) {
                    if (tail0) st->step += 1;
                    st->tail_pending = 1u;
                }
                if (loop) {
                    sy->more = more;
                    __threadfence();
                    atomicAdd(&sy->gen, 1u);
                }
                s_more = more;
            } else {
                s_more = !last_step && gm_wait_generation(&sy->gen, gen, st) && gm_ld_acquire(&sy->more) != 0;
            }
            __threadfence();
        }
        if (!loop) return;
        __syncthreads();
        if (!s_more) return;
    }
}

__global__ void step_begin_kernel(StepSync *sy, unsigned fresh, long long todo) {
    StepSync z{};
    z.fresh = fresh;
    z.todo = todo;
    *sy = z;
}

using StepKernel = void (*)(ForceArgs, StepArgs, PackArgs);

// Shared memory of a block without an opt-in.
constexpr size_t kSharedLimit = 48 * 1024;
// The QUAD kernels' static shared memory (quad_phase's s_e, the barrier's and
// the step's words: 1,024 and 16 bytes), rounded up.
constexpr size_t kQuadStatic = 2048;
static_assert(sizeof(double) * kStepThreads + 256 <= kQuadStatic, "quad_phase's energies");

size_t table_bytes(const ForceArgs &fa) { return sizeof(float4) * (size_t)fa.ntypes * fa.ntypes; }

// A batch reads its [system][type][type] tables through L1, as does a single
// system whose table passes 48 KB.
bool global_table(const ForceArgs &fa) { return fa.e_sys != nullptr || table_bytes(fa) > kSharedLimit; }

// A small system's block per pair item, where its table leaves room for the
// kernel's own shared memory (up to 54 types; with 55 the table alone fits).
bool quad_form(const ForceArgs &fa) {
    return fa.quad && !global_table(fa) && table_bytes(fa) + kQuadStatic <= kSharedLimit;
}

template <bool STEP>
StepKernel pick(const ForceArgs &fa, bool gtab) {
#define GM_STEPK(P, Q, B, M, D) return step_persistent_kernel<P, Q, B, M, STEP, D>
#define GM_STEPB(P, Q, M) { if (gtab) GM_STEPK(P, Q, true, M, false); else if (quad_form(fa)) GM_STEPK(P, Q, false, M, true); \
                            else GM_STEPK(P, Q, false, M, false); }
#define GM_STEPQ(P, M) { if (fa.coulomb) GM_STEPB(P, true, M) else GM_STEPB(P, false, M) }
    if (fa.bonded_mi) GM_STEPQ(true, true)
    if (fa.periodic) GM_STEPQ(true, false)
    GM_STEPQ(false, false)
#undef GM_STEPQ
#undef GM_STEPB
#undef GM_STEPK
}

}  // namespace

bool gm_step_loops(const ForceArgs &fa) { return quad_form(fa); }

int gm_step_persistent_blocks(const ForceArgs &fa) {
    const bool gtab = global_table(fa);
    const size_t smem = gtab ? 0 : table_bytes(fa);
    int dev = 0, sms = 0, per_sm = 0, per_sm_forces = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, pick<true>(fa, gtab), kStepThreads, smem) != cudaSuccess)
        return 0;
    // the force phase alone has more static shared memory than the step
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm_forces, pick<false>(fa, gtab), kStepThreads, smem) !=
            cudaSuccess || per_sm_forces == 0)
        return 0;
    // no more blocks than the tickets (a warp each, a block with quad) or the atoms fill: a
    // small system's barrier waits for fewer arrivals
    const bool quad = quad_form(fa);
    const int chunk = quad ? kStepThreads : ticket_terms<true>(fa), warps = quad ? 1 : kStepThreads / 32;
    const long long tickets = (long long)fa.n_groups * fa.split + bonded_tickets(fa, chunk) + pair14_tickets(fa, chunk);
    const long long fill = (tickets + warps - 1) / warps, atoms = ((long long)fa.n * (quad ? 4 : 1) + kStepThreads - 1) / kStepThreads;
    const long long want = fill > atoms ? fill : atoms;
    return (int)(want < (long long)per_sm * sms ? (want > 0 ? want : 1) : (long long)per_sm * sms);
}

void gm_launch_step_persistent(const ForceArgs &fa, const StepArgs &sa, const PackArgs &pk, int blocks,
                               cudaStream_t s) {
    const bool gtab = global_table(fa);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3(kStepThreads);
    cfg.dynamicSmemBytes = gtab ? 0 : table_bytes(fa);
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, pick<true>(fa, gtab), fa, sa, pk);
}

void gm_launch_forces_persistent(const ForceArgs &fa, StepSync *sync, int blocks, cudaStream_t s) {
    const bool gtab = global_table(fa);
    StepArgs sa{};
    sa.sync = sync;
    PackArgs pk{};
    pick<false>(fa, gtab)<<<blocks, kStepThreads, gtab ? 0 : table_bytes(fa), s>>>(fa, sa, pk);
}

void gm_launch_step_begin(StepSync *sync, bool fresh, long long todo, cudaStream_t s) {
    step_begin_kernel<<<1, 1, 0, s>>>(sync, fresh ? 1u : 0u, todo);
}
