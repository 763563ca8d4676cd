// gm_list.cu — Verlet list build on the device (neighbor.rs:8-55 semantics),
// for one system or a batch of independent systems in one context.
//
// Pipeline at each rebuild (all on the context's stream, no host sync):
//   wrap (periodic only) -> bbox partials -> grid setup -> cell assignment +
//   counting-sort histogram -> scan -> scatter -> in-cell rank by caller
//   index (deterministic order) -> pack -> list build.
// Every kernel runs over all systems at once (blockIdx.y = system) and skips
// the systems whose rebuild flag is clear, so a batch rebuilds only the
// systems that need it.  Each system owns a range of atoms, a 32-aligned
// range of sorted slots (padding slots have perm = -1 and no list), a range
// of cells and its own grid; perm and the list entries hold global indices.
// The list build gives a block 32 consecutive cell-sorted atoms of one system
// and each of its warps one z layer of their candidate cell box (or a share of a
// layer's y rows); the warp streams the candidates near the 32 atoms through
// shared memory, each lane tests them against its own atom and stages what it
// accepts as bits, and the block writes them into the lanes' columns.  The
// test runs in FP32 on hi+lo coordinates; candidates within `margin` of the
// list radius are re-decided with the reference's exact FP64 expression
// (min-image, then dx*dx + dy*dy + dz*dz, no fused multiply-add), so the pair
// set equals the reference's bit for bit.
#include <algorithm>
#include <cfloat>
#include <climits>

#include "gm_internal.cuh"

namespace {


__device__ __forceinline__ double exact_wrap(double x, double L) {
    // neighbor.rs:86-88: x - L * floor(x / L); x itself inside the box (0 <= x <
    // L by its bits, so the quotient rounds below 1; -0.0 goes the long way)
    if ((unsigned long long)__double_as_longlong(x) < (unsigned long long)__double_as_longlong(L)) return x;
    return __dsub_rn(x, __dmul_rn(L, floor(__ddiv_rn(x, L))));
}

// Atom range of system blockIdx.y, or false when it keeps its list.
__device__ __forceinline__ bool sys_atoms(const ListArgs &a, int &a0, int &a1) {
    const int s = blockIdx.y;
    if (!a.sys_flag[s]) return false;
    a0 = a.sys_atom_off[s];
    a1 = a.sys_atom_off[s + 1];
    return true;
}

__global__ void set_flags_kernel(ListArgs a) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s < a.n_sys) a.sys_flag[s] = 1u;
}

__global__ void clear_flags_kernel(ListArgs a) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s < a.n_sys) a.sys_flag[s] = 0u;
    if (s == 0) a.status->rebuild = 0u;
}

// `done` (or nullptr): systems that are wrapped already.
__global__ void wrap_kernel(ListArgs a, double *pos, const unsigned int *done) {
    int a0, a1;
    if (!sys_atoms(a, a0, a1) || (done && done[blockIdx.y])) return;
    const int n = a.n;
    for (int i = a0 + blockIdx.x * blockDim.x + threadIdx.x; i < a1; i += gridDim.x * blockDim.x) {
        pos[i] = exact_wrap(pos[i], a.box[0]);
        pos[n + i] = exact_wrap(pos[n + i], a.box[1]);
        pos[2 * n + i] = exact_wrap(pos[2 * n + i], a.box[2]);
    }
}

// Partial-sum blocks of a system's bbox: as many as a context holding only
// that system uses, so a system's grid (and its FP32 copies) come out the
// same alone or in a batch.
__device__ __forceinline__ int bbox_blocks_of(int n_atoms, int cap) {
    const int b = (n_atoms + 255) / 256;
    return b < 1 ? 1 : (b > cap ? cap : b);
}

// sm[0..8][t], t < width (a power of two): minima, maxima and sums over t, three
// rows each, into column 0.  A level's 9 * k combinations are spread over the
// block: an FP64 instruction holds its scheduler for 64 cycles whatever the
// number of lanes, and with nine of them one after the other in every thread
// the tree of 256 was 72 in a row (15 now).
__device__ __forceinline__ void bbox_tree(double (*sm)[256], int width) {
    for (int k = width / 2; k > 0; k >>= 1) {
        for (int e = threadIdx.x; e < 9 * k; e += blockDim.x) {
            const int v = e / k, t = e - v * k;
            const double x = sm[v][t], y = sm[v][t + k];
            sm[v][t] = v < 3 ? fmin(x, y) : (v < 6 ? fmax(x, y) : x + y);
        }
        __syncthreads();
    }
}

// Per block and system: min x,y,z, max x,y,z and the sum x,y,z.
__global__ void bbox_kernel(ListArgs a) {
    __shared__ double sm[9][256];
    double mn[3] = {DBL_MAX, DBL_MAX, DBL_MAX}, mx[3] = {-DBL_MAX, -DBL_MAX, -DBL_MAX}, sum[3] = {0, 0, 0};
    int a0, a1;
    if (!sys_atoms(a, a0, a1)) return;  // uniform per block
    const int nb = bbox_blocks_of(a1 - a0, 256);
    if ((int)blockIdx.x >= nb) return;
    const int n = a.n;
    for (int i = a0 + blockIdx.x * blockDim.x + threadIdx.x; i < a1; i += nb * blockDim.x) {
        for (int d = 0; d < 3; d++) {
            double v = a.pos[d * n + i];
            mn[d] = fmin(mn[d], v);
            mx[d] = fmax(mx[d], v);
            if (v == v) sum[d] += v;
        }
    }
    for (int d = 0; d < 3; d++) {
        sm[d][threadIdx.x] = mn[d];
        sm[3 + d][threadIdx.x] = mx[d];
        sm[6 + d][threadIdx.x] = sum[d];
    }
    __syncthreads();
    bbox_tree(sm, 256);
    if (threadIdx.x < 9)
        a.bbox_scratch[((size_t)blockIdx.y * a.bbox_blocks + blockIdx.x) * 9 + threadIdx.x] = sm[threadIdx.x][0];
}

// One block per system: reduce its bbox partials, then lay out its grid, a
// dimension per lane (the FP64 divisions are most of the kernel: 1,536 atoms
// 11.9 us with one thread for the three, 4.9 now).
__global__ void __launch_bounds__(256) grid_kernel(ListArgs a, int blocks) {
    const int sys = blockIdx.x;
    if (!a.sys_flag[sys]) return;
    __shared__ double red[9][256];
    __shared__ int s_ncell;
    if (!a.periodic) {
        const double *partial = a.bbox_scratch + (size_t)sys * blocks * 9;
        const int nb = bbox_blocks_of(a.sys_atom_off[sys + 1] - a.sys_atom_off[sys], 256);
        int width = 1;
        while (width < nb) width *= 2;
        if (threadIdx.x < width)
            for (int v = 0; v < 9; v++)
                red[v][threadIdx.x] = threadIdx.x < nb ? partial[threadIdx.x * 9 + v]
                                                       : (v < 3 ? DBL_MAX : (v < 6 ? -DBL_MAX : 0.0));
        __syncthreads();
        bbox_tree(red, width);
    }
    if (threadIdx.x < 32) {
        const unsigned full = 0xffffffffu;
        const int d = min((int)threadIdx.x, 2);
        const bool mine = threadIdx.x < 3;
        GridInfo *g = a.grid + sys;
        const int n_atoms = a.sys_atom_off[sys + 1] - a.sys_atom_off[sys];
        const int max_cells = a.sys_cell_off[sys + 1] - a.sys_cell_off[sys] - 1;
        const double box = a.box[d];
        const double wmin = a.r_list * 0.5 * (1.0 + 1e-5) + 1e-6;
        int nc;
        double lo, origin;
        if (a.periodic) {
            nc = (int)floor(box / wmin);
            if (nc < 1) nc = 1;
            origin = 0.5 * box;
            lo = -0.5 * box;
        } else {
            double mn = red[d][0], mx = red[3 + d][0], sum = red[6 + d][0];
            // The grid covers a core cube around the mean position, at the finest
            // cell width the allocation allows; atoms outside it (evaporated atoms
            // of a droplet in vacuum) are clamped into the edge cells.  Clamping is
            // 1-Lipschitz on cell indices, so the 5x5x5 stencil still finds every
            // pair, and a few outliers no longer coarsen the whole grid.
            const int per_dim = (int)floor(cbrt((double)max_cells));
            double ext = mx - mn;
            if (!(ext == ext) || mx < mn) { ext = 0.0; mn = mx = 0.0; sum = 0.0; }
            // min-image of the reference folds pairs farther apart than box/2;
            // the cell search assumes it never does
            if (mine && ext + a.r_list >= 0.5 * box) atomicOr(&a.status->error, (unsigned)GM_DEV_EXTENT);
            const double mean = n_atoms > 0 ? sum / n_atoms : 0.0;
            const double half = 0.5 * per_dim * wmin;
            double lo_c = fmax(mn, mean - half), hi_c = fmin(mx, mean + half);
            if (!(hi_c >= lo_c)) { lo_c = mn; hi_c = mx; }
            const double pad = 1e-3 * (1.0 + (hi_c - lo_c));
            origin = 0.5 * (lo_c + hi_c);
            lo = (lo_c - origin) - pad;
            nc = (int)floor((hi_c - lo_c + 2.0 * pad) / wmin);
            if (nc < 1) nc = 1;
        }
        // keep the cell count within the allocation by coarsening the grid
        // (coarser cells only widen the 5x5x5 search, never miss a pair)
        int n0, n1, n2;
        for (;;) {
            n0 = __shfl_sync(full, nc, 0), n1 = __shfl_sync(full, nc, 1), n2 = __shfl_sync(full, nc, 2);
            const long long cells = (long long)n0 * n1 * n2;
            if (cells <= max_cells || cells == 1) break;
            nc = nc > 1 ? (nc * 3) / 4 : 1;
        }
        if (mine) {
            const double span = a.periodic ? box : -2.0 * lo;
            const double w = span / nc;
            g->box[d] = (float)box;
            g->inv_box[d] = (float)(1.0 / box);
            g->origin[d] = origin;
            g->nc[d] = nc;
            g->lo[d] = (float)lo;
            g->inv_w[d] = (float)(1.0 / w);
            g->full[d] = a.periodic && nc < 5;
        }
        if (threadIdx.x == 0) {
            g->periodic = a.periodic;
            g->ncell = n0 * n1 * n2;  // <= max_cells by construction
            if (a.sys_far) a.sys_far[sys] = 0u;  // (the static build keeps no list)
            atomicAdd(&a.status->n_rebuilds, 1ull);
            s_ncell = min(n0 * n1 * n2, max_cells);
        }
    }
    // the cells the new grid uses (the only ones assign and the scan touch)
    __syncthreads();
    const int c0 = a.sys_cell_off[sys];
    for (int c = c0 + threadIdx.x; c < c0 + s_ncell; c += blockDim.x) {
        a.cell_count[c] = 0;
        a.cell_cursor[c] = 0;
    }
}


__device__ __forceinline__ int cell_coord(float h, float lo, float inv_w, int nc) {
    float t = floorf((h - lo) * inv_w);
    int c = (int)t;  // NaN converts to 0
    return c < 0 ? 0 : (c >= nc ? nc - 1 : c);
}

__global__ void assign_kernel(ListArgs a) {
    int a0, a1;
    if (!sys_atoms(a, a0, a1)) return;
    const GridInfo *g = a.grid + blockIdx.y;
    const int coff = a.sys_cell_off[blockIdx.y];
    const int max_cells = a.sys_cell_off[blockIdx.y + 1] - coff - 1;
    const int n = a.n;
    for (int i = a0 + blockIdx.x * blockDim.x + threadIdx.x; i < a1; i += gridDim.x * blockDim.x) {
        int c3[3];
        for (int d = 0; d < 3; d++) {
            double x = a.pos[d * n + i];
            a.ref[d * n + i] = x;  // NeighborList::ref_{x,y,z} (neighbor.rs:48-50)
            c3[d] = cell_coord((float)(x - g->origin[d]), g->lo[d], g->inv_w[d], g->nc[d]);
        }
        int c = (c3[2] * g->nc[1] + c3[1]) * g->nc[0] + c3[0];
        if (c < 0 || c >= max_cells) {
            atomicOr(&a.status->error, (unsigned)GM_DEV_CELL_OVERFLOW);
            c = 0;
        }
        a.cell_of[i] = c;
        atomicAdd(&a.cell_count[coff + c], 1);
    }
}

// Exclusive scan of one value per thread over a block (a multiple of 32
// threads, at most 1024), with the block total.
__device__ __forceinline__ int block_exclusive_scan(int v, int *warp_sums, int &total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int x = v;
    for (int o = 1; o < 32; o <<= 1) {
        int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[w] = x;
    __syncthreads();
    if (w == 0) {
        const int nw = blockDim.x >> 5;
        int t = lane < nw ? warp_sums[lane] : 0;
        for (int o = 1; o < 32; o <<= 1) {
            int y = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += y;
        }
        warp_sums[lane] = t;
    }
    __syncthreads();
    const int excl = x - v + (w > 0 ? warp_sums[w - 1] : 0);
    total = warp_sums[(blockDim.x >> 5) - 1];
    __syncthreads();
    return excl;
}

__device__ __forceinline__ int sys_ncell(const ListArgs &a, int s) {
    const int max_cells = a.sys_cell_off[s + 1] - a.sys_cell_off[s] - 1;
    return min(a.grid[s].ncell, max_cells);
}

// Exclusive scan of each system's cell counts into cell_start[0..ncell], one
// block per system walking its cells in chunks of 4096 with a running carry
// (a few chunks for the grids of these systems).
__global__ void __launch_bounds__(1024) scan_cells_kernel(ListArgs a) {
    __shared__ int warp_sums[32];
    const int s = blockIdx.x;
    if (!a.sys_flag[s]) return;
    const int ncell = sys_ncell(a, s), coff = a.sys_cell_off[s];
    int carry = 0;
    for (int base = 0; base <= ncell; base += 4 * (int)blockDim.x) {
        const int i0 = base + 4 * (int)threadIdx.x;
        int v[4], sum = 0;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            v[k] = i0 + k < ncell ? a.cell_count[coff + i0 + k] : 0;
            sum += v[k];
        }
        int total;
        int run = carry + block_exclusive_scan(sum, warp_sums, total);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            if (i0 + k <= ncell) a.cell_start[coff + i0 + k] = run;
            run += v[k];
        }
        carry += total;
    }
}



__global__ void scatter_kernel(ListArgs a) {
    int a0, a1;
    if (!sys_atoms(a, a0, a1)) return;
    const int coff = a.sys_cell_off[blockIdx.y], soff = a.sys_slot_off[blockIdx.y];
    for (int i = a0 + blockIdx.x * blockDim.x + threadIdx.x; i < a1; i += gridDim.x * blockDim.x) {
        const int c = a.cell_of[i];
        const int slot = a.cell_start[coff + c] + atomicAdd(&a.cell_cursor[coff + c], 1);
        a.tmp_atom[soff + slot] = i - a0;
    }
}

// Within a cell, atoms are ordered by caller index: the rank of an atom is
// the number of cell members with a smaller index.  Independent of the
// atomic order of the scatter, so the sorted layout is deterministic.
__global__ void rank_kernel(ListArgs a) {
    int a0, a1;
    if (!sys_atoms(a, a0, a1)) return;
    const int coff = a.sys_cell_off[blockIdx.y], soff = a.sys_slot_off[blockIdx.y];
    const int ns = a1 - a0;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < ns; k += gridDim.x * blockDim.x) {
        const int at = a.tmp_atom[soff + k];
        const int c = a.cell_of[a0 + at];
        const int s0 = a.cell_start[coff + c], s1 = a.cell_start[coff + c + 1];
        if (s1 - s0 > 65536) {
            // no physical system packs this many atoms into one half cell; keep
            // the quadratic rank bounded and report it
            atomicOr(&a.status->error, (unsigned)GM_DEV_CELL_OVERFLOW);
            a.perm[soff + k] = a0 + at;
            a.cell_sorted[soff + k] = c;
            if (a.slot_of) a.slot_of[a0 + at] = soff + k;
            continue;
        }
        int rank = 0;
        for (int m = s0; m < s1; m++) rank += a.tmp_atom[soff + m] < at;
        a.perm[soff + s0 + rank] = a0 + at;
        a.cell_sorted[soff + s0 + rank] = c;
        if (a.slot_of) a.slot_of[a0 + at] = soff + s0 + rank;
    }
}

// Every slot of every system, every force evaluation: the slot records
// relative to the system's grid origin, and the force accumulators cleared.
__global__ void pack_kernel(ListArgs a, bool fp64) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= a.n_slots) return;
    const int at = a.perm[s];
    if (at < 0) return;  // padding slot
    const int n = a.n;
    const GridInfo *g = a.grid + a.atom_sys[at];
    const double x = a.pos[at], y = a.pos[n + at], z = a.pos[2 * n + at];
    gm_pack_record(a.coord + 2 * s, x - g->origin[0], y - g->origin[1], z - g->origin[2], a.qw[at]);
    if (fp64) {
        a.pos64s[s] = make_double4(x, y, z, a.charge64[at]);
        a.type_sorted[s] = a.type[at];
    }
    a.force[at] = 0;
    a.force[n + at] = 0;
    a.force[2 * n + at] = 0;
}

struct Range { int lo, hi, nc, wrap; };

__device__ __forceinline__ Range dim_range(int mn, int mx, int nc, int periodic, int full) {
    Range r;
    r.nc = nc;
    if (full) { r.lo = 0; r.hi = nc - 1; r.wrap = 0; return r; }
    r.lo = mn - 2;
    r.hi = mx + 2;
    if (periodic) {
        if (r.hi - r.lo + 1 >= nc) { r.lo = 0; r.hi = nc - 1; r.wrap = 0; }
        else r.wrap = 1;
    } else {
        r.lo = r.lo < 0 ? 0 : r.lo;
        r.hi = r.hi >= nc ? nc - 1 : r.hi;
        r.wrap = 0;
    }
    return r;
}

__device__ __forceinline__ int wrapi(int c, int nc) { return c < 0 ? c + nc : (c >= nc ? c - nc : c); }

// FP32 squared distance of a staged candidate from the lane's atom (both
// relative to the group's first atom), with the periodic image; every
// product-sum is an explicit FMA, so the candidate test and the bucket of an
// accepted candidate see the same value.
template <bool PERIODIC>
__device__ __forceinline__ float rel_r2(float4 c, float mx, float my, float mz, const GridInfo &g) {
    float dx = c.x - mx, dy = c.y - my, dz = c.z - mz;
    if (PERIODIC) {
        dx = fmaf(-g.box[0], rintf(dx * g.inv_box[0]), dx);
        dy = fmaf(-g.box[1], rintf(dy * g.inv_box[1]), dy);
        dz = fmaf(-g.box[2], rintf(dz * g.inv_box[2]), dz);
    }
    return fmaf(dz, dz, fmaf(dy, dy, dx * dx));
}

// A float as an integer of the same order, for the warp's integer min / max
// reductions (and back: the map is its own inverse).
__device__ __forceinline__ int ordered_int(float v) {
    const int b = __float_as_int(v);
    return b >= 0 ? b : b ^ 0x7fffffff;
}
__device__ __forceinline__ float warp_min(float v) {
    const int r = __reduce_min_sync(0xffffffffu, ordered_int(v));
    return __int_as_float(r >= 0 ? r : r ^ 0x7fffffff);
}
__device__ __forceinline__ float warp_max(float v) {
    const int r = __reduce_max_sync(0xffffffffu, ordered_int(v));
    return __int_as_float(r >= 0 ? r : r ^ 0x7fffffff);
}

// Distance of |d| beyond a half extent h, squared.
__device__ __forceinline__ float beyond2(float d, float h) {
    const float e = fmaxf(fabsf(d) - h, 0.f);
    return e * e;
}

// Candidates a warp holds in shared memory between two rounds of tests (as
// many bytes as a quarter as many staged words).
constexpr int kRound = 256, kRoundY = 64;
// Rows of 32 ints that 32 candidates (a word) take in the staging buffer: their
// slots, then each lane's accept mask and the two bits of its bucket masks.
constexpr int kWordRows = 4;
// gmax of a group whose words did not fit the staging area
constexpr int kStageOver = -1;
// Groups up to which a build splits a layer's y rows over warps: 48 groups 66 us
// against 144, 162 groups 125 against 191, 252 (four systems of 2,000 atoms) 116
// against 135; 256 (16 of 500) 103 against 91, 500 (two of 8,000) 238 against
// 185, 3,072 groups 921 against 793 (partly filled words).
constexpr int kYSplitGroups = 300;

// One block per group, one warp per z layer: warp `seg` tests the candidates
// of z layer `seg` of each row box its lanes need and stages what each lane
// accepts; the block then writes the layers, one after the other, into each
// lane's list column.
//   * The candidates of the row box (5 x 5 x (span + 4) cells) pass 32 at a
//     time, one a lane, and only those within the list radius of the lanes'
//     bounding box are kept, in order, up to 256 in shared memory: 40 % of a
//     row box is out of every lane's reach, and each candidate kept out saves
//     32 distance tests.
//   * Every lane tests the round's candidates, 32 a word, without a branch:
//     an accept bit and the two bits of the distance bucket.  Bits near the
//     list radius (decided in FP64) and pairs as close as the lane's farthest
//     exclusion are looked at one by one; there are few.  A round with no
//     candidate across a face takes no periodic image.
//   * A system of few groups splits each layer into its five y rows as well
//     (YS = 5: 25 warps per group, in the same order): its build is the time
//     of one warp.
//   * The words (not the entries) are staged, coalesced, and their bits counted
//     per bucket; when every layer's counts are known each lane walks its own
//     bits, eight words at a time, and stores each entry once, in its place.
// Bound: issue.  98,304 atoms of water: 800 us; 1,800 us with a test of every
// candidate of the row boxes, a walk per 32 candidates and every entry staged
// (1.5 GB of DRAM traffic).
// Each lane's column is written in distance-bucket order (GM_NBUCKET buckets
// of the build-time distance, bounds in bucket_r2): inside the switch radius,
// the switch band, the shell beyond the cutoff.  Within a bucket the entries
// keep the single-warp sweep order.  The pair kernel's lanes then meet the
// same kind of pair at the same entry and branch together.
//   * A warp that meets more words than its staging area holds (the area is
//     sized from the mean density and the first lists, and a resident run
//     cannot grow it) marks its group; the kernel after it (AGAIN) sweeps a
//     marked group twice instead, to count and to write, in the same order.
template <bool PERIODIC, int YS, bool AGAIN>
__device__ __forceinline__ void build_group(const ListArgs &a, int group, float rl2_lo, float rl2_hi, double rl2_64,
                                            float3 bucket_r2) {
    // the round's candidates: coordinates relative to the group's first atom
    // (FP32; the rounding, under 1e-5 A for candidates within a few list
    // radii, stays far inside the FP64 re-decision margin) and slot; the
    // words being written out in the second part
    constexpr int NSEG = GM_NSEG * YS, ROUND = YS == 1 ? kRound : kRoundY;
    __shared__ float4 s_rel[NSEG][ROUND];
    __shared__ int s_cnt[NSEG][GM_NBUCKET][32];
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int seg = wib;
    const int gseg = group * NSEG + seg;
    if (group * 32 >= a.n_slots) return;
    const int sys = a.group_sys[group];
    if (!a.sys_flag[sys]) return;  // block-uniform: the system keeps its list
    if (AGAIN && a.gmax[group] != kStageOver) return;
    const int soff = a.sys_slot_off[sys], coff = a.sys_cell_off[sys];
    const int ns = a.sys_atom_off[sys + 1] - a.sys_atom_off[sys];
    const int s = group * 32 + lane;
    const bool valid = s - soff < ns;
    const GridInfo g = a.grid[sys];
    const int n = a.n;
    const int cap = a.cap;
    const int *__restrict__ cell_start = a.cell_start + coff;
    // the reference point: the group's first slot (always an atom: systems
    // start on a group boundary)
    float4 rh, rl;
    gm_ld_coord(a.coord + 2 * group * 32, rh, rl);
    float mx = 0.f, my = 0.f, mz = 0.f;
    int my_orig = -1, my_cell = 0;
    if (valid) {
        float4 mh, ml;
        gm_ld_coord(a.coord + 2 * s, mh, ml);
        mx = (mh.x - rh.x) + (ml.x - rl.x);
        my = (mh.y - rh.y) + (ml.y - rl.y);
        mz = (mh.z - rh.z) + (ml.z - rl.z);
        my_orig = a.perm[s];
        my_cell = a.cell_sorted[s];
    }
    // own exclusions as slots, up to 8 kept in registers, and the largest
    // squared distance among them: pairs beyond it skip the scan.  The atom
    // itself (distance 0) is no candidate either.
    int e0 = 0, e1 = 0;
    int ex[8];
    if (valid) { e0 = a.excl_start[my_orig]; e1 = a.excl_start[my_orig + 1]; }
    const int ne = e1 - e0;
    float ex_r2 = 0.f;
    for (int k = 0; k < ne; k++) {
        float4 ch, cl;
        gm_ld_coord(a.coord + 2 * a.slot_of[a.excl[e0 + k]], ch, cl);
        const float4 c = make_float4((ch.x - rh.x) + (cl.x - rl.x), (ch.y - rh.y) + (cl.y - rl.y),
                                     (ch.z - rh.z) + (cl.z - rl.z), 0.f);
        ex_r2 = fmaxf(ex_r2, rel_r2<PERIODIC>(c, mx, my, mz, g));
    }
#pragma unroll
    for (int k = 0; k < 8; k++) ex[k] = k < ne ? a.slot_of[a.excl[e0 + k]] : s;
    // Candidate regions, one per distinct cell row (cy, cz) among the lanes:
    // a group of 32 sorted atoms usually lies in one row of cells, sometimes
    // straddles the end of a row.  Sweeping each row's own 5 x 5 x (span + 4)
    // box keeps the regions tight (one box over both rows would cover the
    // whole row); a lane tests only the candidates of one box, so it never
    // meets a candidate twice.  This warp takes z layer `seg` (and with YS a
    // share of its y rows) of each box.
    const int cx = my_cell % g.nc[0], cy = (my_cell / g.nc[0]) % g.nc[1], cz = my_cell / (g.nc[0] * g.nc[1]);
    const int row_id = valid ? cz * g.nc[1] + cy : -1;
    const int cap_words = a.cap_seg / (YS * kWordRows);
    int *stage = a.stage + (size_t)gseg * cap_words * (kWordRows * 32) + lane;
    int n_words = 0;                    // words met (staged while they fit)
    int nb[GM_NBUCKET] = {0, 0, 0, 0};  // accepted entries per bucket
    const double bx[3] = {a.box[0], a.box[1], a.box[2]};
    const float slack = 1e-3f + (PERIODIC ? 2e-7f * fmaxf(g.box[0], fmaxf(g.box[1], g.box[2])) : 0.f);
    int *my_list = a.list + (size_t)group * 32 * cap + lane;
    int off[GM_NBUCKET];
    int total = 0, inner = 0;  // inner: without the last bucket
    for (int pass = 0;; pass++) {  // one sweep, or with AGAIN two
        unsigned remaining = __ballot_sync(full, valid);
        while (remaining) {
            const int leader = __ffs(remaining) - 1;
            const int R = __shfl_sync(full, row_id, leader);
            bool mine = valid && row_id == R;
            int ymin = R % g.nc[1], ymax = ymin;
            const int zR = R / g.nc[1];
            int xmin, xmax;
            if (!PERIODIC) {
                // Near a droplet's surface 32 atoms may lie in many short rows of
                // one layer: one sweep over all of them when it visits fewer cells
                // (a row's own box is about 5 x 6 cells).  Candidates keep their
                // order; the extra ones are out of reach of the lanes they are
                // new to.
                const bool layer = valid && cz == zR && ((remaining >> lane) & 1u);
                const unsigned peers = __match_any_sync(full, layer ? row_id : -1 - lane);
                const int rows = __popc(__ballot_sync(full, layer && (peers & ((1u << lane) - 1u)) == 0));
                ymin = __reduce_min_sync(full, layer ? cy : INT_MAX);
                ymax = __reduce_max_sync(full, layer ? cy : INT_MIN);
                xmin = __reduce_min_sync(full, layer ? cx : INT_MAX);
                xmax = __reduce_max_sync(full, layer ? cx : INT_MIN);
                if (rows > 1 && ymax - ymin < 28 && (xmax - xmin + 5) * (ymax - ymin + 5) <= 30 * rows) mine = layer;
                else ymin = ymax = R % g.nc[1];
            }
            remaining &= ~__ballot_sync(full, mine);
            xmin = __reduce_min_sync(full, mine ? cx : INT_MAX);
            xmax = __reduce_max_sync(full, mine ? cx : INT_MIN);
            Range rx = dim_range(xmin, xmax, g.nc[0], g.periodic, g.full[0]);
            Range ry = dim_range(ymin, ymax, g.nc[1], g.periodic, g.full[1]);
            Range rz = dim_range(zR, zR, g.nc[2], g.periodic, g.full[2]);
            if (YS > 1) {
                const int per = (ry.hi - ry.lo + YS) / YS;
                ry.lo += seg % YS * per;
                ry.hi = min(ry.hi, ry.lo + per - 1);
            }
            const int zz = rz.lo + seg / YS;
            if (zz > rz.hi || ry.lo > ry.hi) continue;  // warp-uniform
            const int z = rz.wrap ? wrapi(zz, g.nc[2]) : zz;
            // the lanes' bounding box
            const float lox = warp_min(mine ? mx : FLT_MAX), hix = warp_max(mine ? mx : -FLT_MAX);
            const float loy = warp_min(mine ? my : FLT_MAX), hiy = warp_max(mine ? my : -FLT_MAX);
            const float loz = warp_min(mine ? mz : FLT_MAX), hiz = warp_max(mine ? mz : -FLT_MAX);
            const float bcx = 0.5f * (lox + hix), bcy = 0.5f * (loy + hiy), bcz = 0.5f * (loz + hiz);
            // half extents, wider by the FP32 roundings of the tests below
            const float bhx = 0.5f * (hix - lox) + slack, bhy = 0.5f * (hiy - loy) + slack, bhz = 0.5f * (hiz - loz) + slack;
            // The x extent of each y row as one or two runs of consecutive cells
            // (at most 32): lane r holds the slots [run_b, run_e) of run r.
            int x0[2], x1[2], nrun = 1;
            x0[0] = rx.lo; x1[0] = rx.hi; x0[1] = 0; x1[1] = -1;
            if (rx.wrap && rx.lo < 0) { x0[0] = rx.lo + g.nc[0]; x1[0] = g.nc[0] - 1; x0[1] = 0; x1[1] = rx.hi; nrun = 2; }
            else if (rx.wrap && rx.hi >= g.nc[0]) { x1[0] = g.nc[0] - 1; x0[1] = 0; x1[1] = rx.hi - g.nc[0]; nrun = 2; }
            const int runs = (ry.hi - ry.lo + 1) * nrun;
            int run_b = 0, run_e = 0;
            if (lane < runs) {
                const int yy = ry.lo + lane / nrun, sg = lane - lane / nrun * nrun;
                const int row = (z * g.nc[1] + (ry.wrap ? wrapi(yy, g.nc[1]) : yy)) * g.nc[0];
                run_b = soff + cell_start[row + x0[sg]];
                run_e = soff + cell_start[row + x1[sg] + 1];
            }
            int run = 0, base = __shfl_sync(full, run_b, 0), end = __shfl_sync(full, run_e, 0);
            int held = 0;               // candidates of the round
            bool image = false;         // periodic: one of them may need the image
            for (;;) {
                while (base >= end && ++run < runs) {
                    base = __shfl_sync(full, run_b, run);
                    end = __shfl_sync(full, run_e, run);
                }
                const bool more = run < runs;
                if (more) {
                    const int t = base + lane;
                    base += 32;
                    float4 c = make_float4(0.f, 0.f, 0.f, __int_as_float(t));
                    bool keep = false, far = false;
                    if (t < end) {
                        float4 ch, cl;
                        gm_ld_coord(a.coord + 2 * t, ch, cl);
                        c.x = (ch.x - rh.x) + (cl.x - rl.x);
                        c.y = (ch.y - rh.y) + (cl.y - rl.y);
                        c.z = (ch.z - rh.z) + (cl.z - rl.z);
                        float dx = c.x - bcx, dy = c.y - bcy, dz = c.z - bcz;
                        if (PERIODIC) {
                            // a raw difference below half the box from every lane
                            // of the bounding box needs no image
                            far = fabsf(dx) + bhx >= 0.49f * g.box[0] || fabsf(dy) + bhy >= 0.49f * g.box[1] ||
                                  fabsf(dz) + bhz >= 0.49f * g.box[2];
                            dx = fmaf(-g.box[0], rintf(dx * g.inv_box[0]), dx);
                            dy = fmaf(-g.box[1], rintf(dy * g.inv_box[1]), dy);
                            dz = fmaf(-g.box[2], rintf(dz * g.inv_box[2]), dz);
                        }
                        keep = beyond2(dx, bhx) + beyond2(dy, bhy) + beyond2(dz, bhz) <= rl2_hi;
                    }
                    const unsigned kept = __ballot_sync(full, keep);
                    if (keep) s_rel[wib][held + __popc(kept & ((1u << lane) - 1u))] = c;
                    held += __popc(kept);
                    if (PERIODIC) image |= __any_sync(full, keep && far);
                }
                if (more && held <= ROUND - 32) continue;
                if (held == 0) break;
                // ---- a round: all lanes test, 32 candidates a word
                __syncwarp();
                for (int w0 = 0; w0 < held; w0 += 32) {
                    unsigned acc = 0, blo = 0, bhi = 0, look = 0;
                    auto test = [&](float r2, int k) {
                        const bool in = r2 <= rl2_hi, far1 = r2 > bucket_r2.y;
                        acc |= (in ? 1u : 0u) << k;
                        bhi |= (far1 ? 1u : 0u) << k;
                        blo |= (r2 > (far1 ? bucket_r2.z : bucket_r2.x) ? 1u : 0u) << k;
                        look |= (in && (r2 > rl2_lo || r2 <= ex_r2) ? 1u : 0u) << k;
                    };
                    if (PERIODIC && image) {
#pragma unroll
                        for (int k = 0; k < 32; k++) test(rel_r2<true>(s_rel[wib][w0 + k], mx, my, mz, g), k);
                    } else {
#pragma unroll
                        for (int k = 0; k < 32; k++) test(rel_r2<false>(s_rel[wib][w0 + k], mx, my, mz, g), k);
                    }
                    const int m = held - w0;
                    const unsigned live = !mine ? 0u : m < 32 ? (1u << m) - 1u : full;
                    acc &= live;
                    look &= live;
                    while (look) {
                        const int k = __ffs(look) - 1;
                        look &= look - 1;
                        const float4 c = s_rel[wib][w0 + k];
                        const int slot = __float_as_int(c.w);
                        const float r2 = rel_r2<PERIODIC>(c, mx, my, mz, g);
                        bool drop = false;
                        if (r2 > rl2_lo) {
                            // the reference's own FP64 decision
                            const int jo = a.perm[slot];
                            double ex_ = gm_min_image(__dsub_rn(a.pos[jo], a.pos[my_orig]), bx[0]);
                            double ey_ = gm_min_image(__dsub_rn(a.pos[n + jo], a.pos[n + my_orig]), bx[1]);
                            double ez_ = gm_min_image(__dsub_rn(a.pos[2 * n + jo], a.pos[2 * n + my_orig]), bx[2]);
                            double rr = __dadd_rn(__dadd_rn(__dmul_rn(ex_, ex_), __dmul_rn(ey_, ey_)), __dmul_rn(ez_, ez_));
                            drop = !(rr <= rl2_64);
                        }
                        if (r2 <= ex_r2) {
                            drop |= slot == s;
#pragma unroll
                            for (int q = 0; q < 8; q++) drop |= ex[q] == slot;
                            for (int q = e0 + 8; q < e1; q++) drop |= a.slot_of[a.excl[q]] == slot;
                        }
                        if (drop) acc &= ~(1u << k);
                    }
                    if (AGAIN && pass == 1) {
                        while (acc) {
                            const int k = __ffs(acc) - 1;
                            acc &= acc - 1;
                            const int bk = ((blo >> k) & 1u) + 2 * ((bhi >> k) & 1u);
                            int pos = 0;
#pragma unroll
                            for (int q = 0; q < GM_NBUCKET; q++) {
                                if (bk == q) { pos = off[q]; off[q]++; }
                            }
                            if (pos < cap) my_list[(size_t)pos * 32] = __float_as_int(s_rel[wib][w0 + k].w);
                        }
                    } else if (AGAIN || n_words < cap_words) {  // (else the group is marked below)
                        nb[0] += __popc(acc & ~(blo | bhi));
                        nb[1] += __popc(acc & blo & ~bhi);
                        nb[2] += __popc(acc & bhi & ~blo);
                        nb[3] += __popc(acc & blo & bhi);
                        if (!AGAIN) {
                            int *row = stage + (size_t)n_words * (kWordRows * 32);
                            row[0] = __float_as_int(s_rel[wib][w0 + lane].w);
                            row[32] = (int)acc;
                            row[64] = (int)blo;
                            row[96] = (int)bhi;
                        }
                    }
                    n_words++;
                }
                __syncwarp();
                held = 0;
                image = false;
                if (!more) break;
            }
        }
        // the layers' entries go into the column one layer after the other
        if (AGAIN && pass == 1) break;
        if (!AGAIN && lane == 0) atomicMax(&a.status->max_layer, (unsigned)(n_words * kWordRows * YS));
        const bool over = !AGAIN && n_words > cap_words;
#pragma unroll
        for (int q = 0; q < GM_NBUCKET; q++) s_cnt[seg][q][lane] = nb[q];
        if (__syncthreads_or(over)) {
            if (threadIdx.x == 0) {
                a.gmax[group] = kStageOver;
                atomicOr(&a.status->stage_over, 1u);
            }
            return;
        }
        // this layer's first position in each bucket: the earlier buckets of all
        // layers, then this bucket of the earlier layers
#pragma unroll
        for (int q = 0; q < GM_NBUCKET; q++) {
            int before = 0, all = 0;
#pragma unroll
            for (int k = 0; k < NSEG; k++) {
                const int ck = s_cnt[k][q][lane];
                before += k < seg ? ck : 0;
                all += ck;
            }
            off[q] = total + before;
            inner = total;
            total += all;
        }
        if (AGAIN) continue;
        constexpr int WB = ROUND / 32;  // words at a time: [row][word][lane]
        int *buf = reinterpret_cast<int *>(s_rel[wib]);
        for (int w0 = 0; w0 < n_words; w0 += WB) {
            const int words = min(WB, n_words - w0);
            __syncwarp();
            const int *row = stage + (size_t)w0 * (kWordRows * 32);
            int v[WB * kWordRows];
#pragma unroll
            for (int k = 0; k < WB * kWordRows; k++) v[k] = k < words * kWordRows ? row[k * 32] : 0;
#pragma unroll
            for (int k = 0; k < WB * kWordRows; k++) buf[((k % kWordRows) * WB + k / kWordRows) * 32 + lane] = v[k];
            __syncwarp();
            int w = 0;
            unsigned acc = (unsigned)buf[WB * 32 + lane], blo = (unsigned)buf[2 * WB * 32 + lane],
                     bhi = (unsigned)buf[3 * WB * 32 + lane];
            for (;;) {
                while (acc == 0 && ++w < words) {
                    acc = (unsigned)buf[(WB + w) * 32 + lane];
                    blo = (unsigned)buf[(2 * WB + w) * 32 + lane];
                    bhi = (unsigned)buf[(3 * WB + w) * 32 + lane];
                }
                if (acc == 0) break;
                const int k = __ffs(acc) - 1;
                acc &= acc - 1;
                const int bk = ((blo >> k) & 1u) + 2 * ((bhi >> k) & 1u);
                int pos = 0;
#pragma unroll
                for (int q = 0; q < GM_NBUCKET; q++) {
                    if (bk == q) { pos = off[q]; off[q]++; }
                }
                if (pos < cap) my_list[(size_t)pos * 32] = buf[w * 32 + k];
            }
        }
        break;
    }
    if (seg == 0) {
        if (valid) {
            a.count[s] = total < cap ? total : cap;
            a.count_in[s] = inner < cap ? inner : cap;
        }
        if (valid && total > cap) atomicOr(&a.status->error, (unsigned)GM_DEV_LIST_OVERFLOW);
        int c = valid ? (total < cap ? total : cap) : 0;
        int tm = valid ? total : 0;
        const int ci = __reduce_max_sync(full, valid ? min(inner, cap) : 0);
        for (int o = 16; o > 0; o >>= 1) {
            c = max(c, __shfl_xor_sync(0xffffffffu, c, o));
            tm = max(tm, __shfl_xor_sync(0xffffffffu, tm, o));
        }
        if (lane == 0) {
            a.gmax[group] = c;
            a.gmax_in[group] = ci;
            atomicMax(&a.status->max_count, (unsigned)tm);
        }
    }
}

template <bool PERIODIC, int YS>
__global__ void __launch_bounds__(GM_NSEG * YS * 32, YS == 1 ? 5 : 1)
build_kernel(ListArgs a, float rl2_lo, float rl2_hi, double rl2_64, float3 bucket_r2) {
    build_group<PERIODIC, YS, false>(a, blockIdx.x, rl2_lo, rl2_hi, rl2_64, bucket_r2);
}

// The groups the build marked (usually none: one read of the status word).
constexpr int kAgainBlocks = 304;
template <bool PERIODIC>
__global__ void __launch_bounds__(GM_NSEG * 32)
build_again_kernel(ListArgs a, float rl2_lo, float rl2_hi, double rl2_64, float3 bucket_r2) {
    if (a.status->stage_over == 0) return;
    for (int group = blockIdx.x; group * 32 < a.n_slots; group += gridDim.x) {
        build_group<PERIODIC, 1, true>(a, group, rl2_lo, rl2_hi, rl2_64, bucket_r2);
        __syncthreads();
    }
}

// Per-system launch shape: x covers the largest system, y the systems.
dim3 sys_grid(const ListArgs &a, int per_block, int cap_blocks) {
    int bx = (a.max_sys_atoms + per_block - 1) / per_block;
    bx = bx < 1 ? 1 : (bx > cap_blocks ? cap_blocks : bx);
    return dim3((unsigned)bx, (unsigned)a.n_sys, 1);
}

}  // namespace

void gm_launch_flags(const ListArgs &a, bool set, cudaStream_t s) {
    if (set) set_flags_kernel<<<(a.n_sys + 255) / 256, 256, 0, s>>>(a);
    else clear_flags_kernel<<<(a.n_sys + 255) / 256, 256, 0, s>>>(a);
}

void gm_launch_wrap(const ListArgs &a, double *pos, const unsigned int *done, cudaStream_t s) {
    if (!a.periodic || a.n == 0) return;
    wrap_kernel<<<sys_grid(a, 256, 4096), 256, 0, s>>>(a, pos, done);
}

void gm_launch_grid(const ListArgs &a, cudaStream_t s) {
    if (!a.periodic && a.n > 0) bbox_kernel<<<dim3((unsigned)a.bbox_blocks, (unsigned)a.n_sys), 256, 0, s>>>(a);
    grid_kernel<<<a.n_sys, 256, 0, s>>>(a, a.bbox_blocks);
}

void gm_launch_bin(const ListArgs &a, cudaStream_t s) {
    // the grid kernel cleared the cells
    if (a.n > 0) assign_kernel<<<sys_grid(a, 256, 4096), 256, 0, s>>>(a);
    scan_cells_kernel<<<a.n_sys, 1024, 0, s>>>(a);
    if (a.n > 0) {
        scatter_kernel<<<sys_grid(a, 256, 4096), 256, 0, s>>>(a);
        rank_kernel<<<sys_grid(a, 256, 4096), 256, 0, s>>>(a);
    }
}

void gm_launch_pack(const ListArgs &a, bool fp64, cudaStream_t s) {
    if (a.n_slots == 0) return;
    pack_kernel<<<(a.n_slots + 255) / 256, 256, 0, s>>>(a, fp64);
}

// A build of every system covers all groups, another of a batch a few systems,
// as many groups as one of them on average: with the average for both the first
// build of 64 systems of 2,000 atoms took 1,323 us (now 709), of 256 of 500 1,235
// (535).
bool gm_build_splits_rows(const ListArgs &a, bool all) {
    const int groups = a.n_slots / 32;
    return (all ? groups : groups / a.n_sys) <= kYSplitGroups;
}

void gm_launch_build(const ListArgs &a, bool all, cudaStream_t s) {
    if (a.n_slots == 0) return;
    const int groups = a.n_slots / 32;
    const double rl2 = a.r_list * a.r_list;  // neighbor.rs:25
    const double margin = 1e-3 * (rl2 > 144.0 ? rl2 / 144.0 : 1.0);
    // bucket bounds: the switch radius, the cutoff, halfway to the list radius
    const double rsh = 0.5 * (a.r_cut + a.r_list);
    const float3 bk = make_float3((float)(a.r_switch * a.r_switch), (float)(a.r_cut * a.r_cut), (float)(rsh * rsh));
    const float lo = (float)(rl2 - margin), hi = (float)(rl2 + margin);
    const bool ysplit = gm_build_splits_rows(a, all);
#define GM_BUILD(P, Y) build_kernel<P, Y><<<groups, GM_NSEG * Y * 32, 0, s>>>(a, lo, hi, rl2, bk)
    if (a.periodic) { if (ysplit) GM_BUILD(true, 5); else GM_BUILD(true, 1); }
    else { if (ysplit) GM_BUILD(false, 5); else GM_BUILD(false, 1); }
#undef GM_BUILD
    const int again = groups < kAgainBlocks ? groups : kAgainBlocks;
    if (a.periodic) build_again_kernel<true><<<again, GM_NSEG * 32, 0, s>>>(a, lo, hi, rl2, bk);
    else build_again_kernel<false><<<again, GM_NSEG * 32, 0, s>>>(a, lo, hi, rl2, bk);
}
