// Verlet pair list on the GPU.
//
// Same pair set as CellManager::update_pair_list (src/utils/CellManager.cpp:
// 216-314) and Ensemble::build_pairlist (src/Ensemble.cpp:492-525): all
// unordered pairs (i, j) not in the exclusion table whose minimum-image FP64
// distance squared, computed as the reference computes it, is below
// (cutoff + cutBuff)^2.  Sites are binned with the reference's cell formula
// (CellManager::find_cell, CellManager.h:75-102, clamping included), and the
// 27-cell stencil around each site's cell is the symmetric closure of the
// reference's own-cell + 13-cell half shell, so the list holds each pair in
// both directions ("full list"): every site's forces are then summed by the
// threads that own it, with no atomics.
//
// The list is rebuilt only when flags[0] is set (the integrate kernel raises
// it when a displacement since the last build exceeds cutBuff/2,
// LFIntegrator.cpp:307-341); every kernel here reads the flag and returns at
// once otherwise, so the step can run as one fixed CUDA graph.  Two kernels
// (one for a box without cells): k_cells bins the sites, k_build writes the
// rows.
#include <cooperative_groups.h>
#include "smd_ctx.cuh"

namespace smd {

namespace cg = cooperative_groups;

constexpr int NB_SITES = LIST_GROUP;   // sites of one cell per group: one warp each in k_build
constexpr int NB_STAGE = 1024;         // candidates staged at a time
constexpr int NB_CELLS = 36;           // stencil cells at most (4 x 3 x 3 under shear)
constexpr int CELL_CTAS = 8, CELL_THREADS = 1024;

// the curve's position of sub-cell x + 4 y + 16 z (Skilling 2004, AIP Conf.
// Proc. 707: 381, two bits per axis)
__constant__ unsigned char HILBERT4[64] = {
     0,  3, 60, 63,  1,  2, 61, 62, 30, 31, 32, 33, 29, 28, 35, 34,
     7,  4, 59, 56,  6,  5, 58, 57, 25, 24, 39, 38, 26, 27, 36, 37,
     8, 11, 52, 55, 15, 12, 51, 48, 16, 23, 40, 47, 19, 20, 43, 44,
     9, 10, 53, 54, 14, 13, 50, 49, 17, 22, 41, 46, 18, 21, 42, 45};

// farther than 0.75 L from the origin on some axis (or not finite)
__device__ __forceinline__ bool far_out(const double4 &p, const Box &b) {
    return !(fabs(p.x) <= 0.75 * b.L[0] && fabs(p.y) <= 0.75 * b.L[1] && fabs(p.z) <= 0.75 * b.L[2]);
}

// sc: the box edges over the ones the grid was laid out for (1 but under
// the barostat, which scales positions and box together)
// (key: the place of the site's sub-cell, 4 x 4 x 4 per cell, on a Hilbert
// curve through them: consecutive keys are neighbours)
__device__ __forceinline__ int ref_cell(const double4 &p, const CellGrid &g, const double (&sc)[3], unsigned &key) {
    int c[3];
    key = 0;
    const double pp[3] = {p.x, p.y, p.z};
#pragma unroll
    for (int d = 0; d < 3; d++) {
        double delta = sc[d] == 1.0 ? pp[d] - g.origin[d] : pp[d] / sc[d] - g.origin[d];
        int x = (int)(delta * g.rlen[d]);
        if (x >= g.n[d]) x = g.n[d] - 1;
        else if (x < 0) x = 0;
        c[d] = x;
        key += (unsigned)min(3, max(0, (int)((delta * g.rlen[d] - x) * 4.0))) << 2 * d;
    }
    key = HILBERT4[key];
    return (c[2] * g.n[1] + c[1]) * g.n[0] + c[0];
}

// Bins the sites: cells by the reference's formula, each cell's sites ordered
// by sub-cell and index (so the list rows, and with them every per-thread
// partial sum, come out the same on every run, and 32 consecutive sites lie
// close together), their box fractions in that order, and the groups of up
// to NB_SITES sites of one cell that k_build's blocks take.  One cluster of
// blocks, which the hardware places together, so the four phases need no
// launches of their own: count, scan (first block), fill, and order (a site's
// rank is the number of smaller keys in its cell).
constexpr int KEY_SHIFT = 25;   // site index bits below the sub-cell key
__global__ void __cluster_dims__(CELL_CTAS, 1, 1) __launch_bounds__(CELL_THREADS)
k_cells(int n, const double4 *__restrict__ pos4, CellGrid g, Box box0, const double *le, int *cell_of,
        unsigned *cell_slot, int *cell_count, int *cell_start, unsigned *cell_fill, int4 *cell_q, int2 *group,
        int *ngroup, int *flags, const Box *dbox) {
    if (!flags[0]) return;   // the same for every block: nothing writes the flag before k_build
    cg::cluster_group cl = cg::this_cluster();
    const int rank = cl.block_rank(), tid = rank * CELL_THREADS + threadIdx.x, all = CELL_CTAS * CELL_THREADS;
    const Box box = dbox ? *dbox : box0;
    double sc[3] = {1.0, 1.0, 1.0};
    if (dbox)
        for (int d = 0; d < 3; d++) sc[d] = box.L[d] / g.L0[d];
    const unsigned low = n <= 1 << KEY_SHIFT ? (1u << KEY_SHIFT) - 1 : 0xffffffffu;   // larger systems: no key
    for (int i = tid; i < n; i += all) {
        unsigned key;
        const double4 p = pos4[i];
        const int c = ref_cell(p, g, sc, key);
        cell_of[i] = c;
        cell_slot[i] = (unsigned)atomicAdd(&cell_count[c], 1) | (low == 0xffffffffu ? 0u : key << KEY_SHIFT);
        if (far_out(p, box)) atomicOr(&flags[5], 1);
    }
    cl.sync();
    if (rank == 0) {
        // exclusive scan of the cells' site counts (low word) and group
        // counts (high word); zeroes the counts for the next build
        __shared__ unsigned long long s_carry, s_warp[32];
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
        if (threadIdx.x == 0) s_carry = 0;
        __syncthreads();
        for (int base = 0; base < g.ncell; base += CELL_THREADS) {
            const int c = base + threadIdx.x;
            const unsigned cnt = c < g.ncell ? (unsigned)__ldcg(&cell_count[c]) : 0u, ng = (cnt + NB_SITES - 1) / NB_SITES;
            const unsigned long long v = (unsigned long long)ng << 32 | cnt;
            unsigned long long x = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned long long y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            if (lane == 31) s_warp[w] = x;
            __syncthreads();
            if (w == 0) {
                unsigned long long s = s_warp[lane];
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const unsigned long long y = __shfl_up_sync(0xffffffffu, s, o);
                    if (lane >= o) s += y;
                }
                s_warp[lane] = s;
            }
            __syncthreads();
            const unsigned long long excl = x - v + (w > 0 ? s_warp[w - 1] : 0) + s_carry;
            if (c < g.ncell) {
                const int start = (int)(unsigned)excl, g0 = (int)(excl >> 32);
                cell_start[c] = start;
                cell_count[c] = 0;
                for (unsigned q = 0; q < ng; q++) group[g0 + q] = make_int2(c, start + q * NB_SITES);
            }
            __syncthreads();
            if (threadIdx.x == CELL_THREADS - 1) s_carry = excl + v;
            __syncthreads();
        }
        if (threadIdx.x == 0) {
            cell_start[g.ncell] = (int)(unsigned)s_carry;
            *ngroup = (int)(s_carry >> 32);
        }
    }
    cl.sync();
    for (int i = tid; i < n; i += all) {
        const unsigned s = cell_slot[i];
        cell_fill[cell_start[cell_of[i]] + (s & low)] = (unsigned)i | (s & ~low);
    }
    cl.sync();
    const double delta = le ? *le : 0.0;
    for (int i = tid; i < n; i += all) {
        const int c = cell_of[i], s = cell_start[c], e = cell_start[c + 1];
        const unsigned me = (unsigned)i | (cell_slot[i] & ~low);
        int r = 0;
#pragma unroll 8
        for (int k = s; k < e; k++) r += cell_fill[k] < me;
        int4 q = site_frac(pos4[i], box, le != nullptr, delta);
        q.w = i;
        cell_q[s + r] = q;
    }
}

struct BuildArgs {
    int n, max_nbr;
    const double4 *pos4;
    double4 *disp4;
    const int *mol, *excl_off, *excl;
    int excl_intermol;  // some exclusion joins two molecules
    int mol_sites;
    const int *cell_start;
    const int4 *cell_q; // the sites in cell order: box fractions, index
    const int2 *group;  // (cell, first slot) of each group, or null without cells
    const int *ngroup;
    CellGrid g;
    Box box;
    double rl2;
    int *nbr, *nnbr;
    unsigned int *status, *ticket;
    int *flags;
    double *le;         // Lees-Edwards offset on the device, or null
    const Box *dbox;    // the box on the device (barostat), or null: box
};

// r^2 of the reference's pair test, without contraction into FMA
// (x86-64 -O2 builds of the reference use separate multiply and add).
__device__ __forceinline__ double ref_r2(const double4 &a, const double4 &b, const Box &bx,
                                         bool pbc, bool le, double delta) {
    double dx = __dsub_rn(b.x, a.x), dy = __dsub_rn(b.y, a.y), dz = __dsub_rn(b.z, a.z);
    if (le) {
        min_image_le(dx, dy, dz, bx, delta);
    } else if (pbc) {
        dx = pbc1(dx, bx.L[0], bx.half[0]);
        dy = pbc1(dy, bx.L[1], bx.half[1]);
        dz = pbc1(dz, bx.L[2], bx.half[2]);
    }
    return __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
}

// The list rows.  A block takes groups of up to NB_SITES sites of one cell
// (without cells: consecutive sites), one warp per site, which share their
// stencil: its candidates, cell by cell in the order dz, dy, dx (without
// cells: every site), are staged NB_STAGE at a time as 32-bit box fractions.
// Each 32 consecutive ones get a bounding box; a warp skips the chunks whose
// box is beyond the list radius of its site (one lane per chunk) and tests
// the others 32 at a time, appending in candidate order (ballot + popc), so
// the row order is deterministic.
//
// The test runs in FP32 on the exact integer minimum image; only a candidate
// within 1e-5 of the list radius (relative, in r^2; the fractions and FP32
// err below 2e-6) takes the reference's FP64 test, so the pair set is the
// reference's.  When some site is farther than 0.75 L from the origin
// (uploaded unwrapped), every candidate takes the FP64 test: the reference's
// minimum image takes a bounded number of steps and none inside a cell,
// which matches the integer one only for sites in or near the box.  That is
// settled before the first test, by k_cells or (without cells) by every block
// for itself, so that both rows of a pair follow the same rule.
// Instruction issue bounds the pass, and most candidates are beyond the
// radius (92 % for water in 3 x 3 x 3 cells), hence the skips.  Against one
// FP64 test per candidate: 6480 sites of water 212 -> 98 us, 12288 sites 340 ->
// 119 us a build; a step without a build 1.5 us (with k_cells 2.7 us in place
// of 8 us for five gated launches).
template <bool LE>
__global__ void __launch_bounds__(NB_SITES * 32, 5) k_build(BuildArgs a) {
    if (!a.flags[0]) return;
    __shared__ int4 s_q[NB_STAGE];       // fractions, site
    __shared__ int s_m[NB_STAGE];        // molecule; bit 31: same cell as the group
    __shared__ float s_lo[3][NB_STAGE / 32], s_hi[3][NB_STAGE / 32];   // chunk boxes about the group's first site
    __shared__ int s_off[NB_CELLS + 1], s_cs[NB_CELLS], s_nc[NB_CELLS];
    __shared__ int4 s_c;                 // the group's first site
    const Box box = a.dbox ? *a.dbox : a.box;
    const double delta = LE ? *a.le : 0.0;
    const unsigned dfrac = LE ? le_frac(delta, box.inv[0]) : 0u;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const float sx = (float)(box.L[0] / 4294967296.0), sy = (float)(box.L[1] / 4294967296.0),
                sz = (float)(box.L[2] / 4294967296.0);
    const int ngroup = a.group ? *a.ngroup : (a.n + NB_SITES - 1) / NB_SITES;
    bool far = false;
    if (a.group) {
        far = a.flags[5];
    } else {
        // eight loads of a thread in flight
#pragma unroll 8
        for (int j = threadIdx.x; j < a.n; j += NB_SITES * 32) far |= far_out(a.pos4[j], box);
        far = __syncthreads_or(far);
    }
    for (int gi = blockIdx.x; gi < ngroup; gi += gridDim.x) {
        const int2 grp = a.group ? a.group[gi] : make_int2(-1, gi * NB_SITES);
        const int c = grp.x;
        __syncthreads();   // the previous group's shared memory is done with
        if (a.group && threadIdx.x < NB_CELLS) {
            const int t = threadIdx.x, dz = t / 12 - 1, dy = (t / 4) % 3 - 1, dx = t % 4 - 1;
            const int cx = c % a.g.n[0], cy = (c / a.g.n[0]) % a.g.n[1], cz = c / (a.g.n[0] * a.g.n[1]);
            int z = cz + dz; z = z < 0 ? z + a.g.n[2] : (z >= a.g.n[2] ? z - a.g.n[2] : z);
            int y = cy + dy;
            // under shear, the images across the y boundary sit delta
            // further in x: the x window moves by delta and widens by a cell
            const int wy = y < 0 ? -1 : (y >= a.g.n[1] ? 1 : 0);
            y = y < 0 ? y + a.g.n[1] : (y >= a.g.n[1] ? y - a.g.n[1] : y);
            int sh = 0, dx1 = 1;
            if (LE && wy != 0) {
                sh = (int)floor((wy < 0 ? delta : -delta) * a.g.rlen[0]);
                dx1 = 2;
            }
            int x = (cx + sh + dx) % a.g.n[0];
            x = x < 0 ? x + a.g.n[0] : x;
            const int nc = (z * a.g.n[1] + y) * a.g.n[0] + x;
            s_nc[t] = nc;
            s_cs[t] = a.cell_start[nc];
            s_off[t + 1] = dx <= dx1 ? a.cell_start[nc + 1] - a.cell_start[nc] : 0;
        }
        const int last = a.group ? a.cell_start[c + 1] : a.n;
        const int slot = grp.y + w;
        int4 fi = make_int4(0, 0, 0, -1);
        if (slot < last) {
            if (a.group) {
                fi = a.cell_q[slot];
            } else {
                fi = site_frac(a.pos4[slot], box, LE, delta);
                fi.w = slot;
            }
        }
        const int i = fi.w;
        int mi = 0, e0 = 0, e1 = 0, count = 0;
        if (i >= 0) {
            mi = a.mol[i];
            e0 = a.excl_off[i];
            e1 = a.excl_off[i + 1];
            if (lane == 0) a.disp4[i] = make_double4(0, 0, 0, 0);
        }
        if (threadIdx.x == 0) s_c = fi;
        __syncthreads();
        if (a.group && threadIdx.x == 0) {
            s_off[0] = 0;
            for (int t = 0; t < NB_CELLS; t++) s_off[t + 1] += s_off[t];
        }
        __syncthreads();
        const int total = a.group ? s_off[NB_CELLS] : a.n;
        const float dix = (float)(fi.x - s_c.x), diy = (float)(fi.y - s_c.y), diz = (float)(fi.z - s_c.z);
        for (int base = 0; base < total; base += NB_STAGE) {
            const int cnt = min(NB_STAGE, total - base), nchunk = (cnt + 31) >> 5;
            __syncthreads();
            // warp w stages the chunks w, w + 8, ... and boxes each about its
            // own first site, so that a chunk across the half-box plane of
            // the group's site keeps its size
            for (int ch = w; ch < nchunk; ch += NB_SITES) {
                const int f = ch * 32 + lane;
                int j = base + min(f, cnt - 1), same = 0;
                int4 q;
                if (a.group) {
                    int t = 0;   // the stencil cell: the last t with s_off[t] <= j
#pragma unroll
                    for (int o = 32; o > 0; o >>= 1)
                        if (t + o < NB_CELLS && s_off[t + o] <= j) t += o;
                    q = a.cell_q[s_cs[t] + j - s_off[t]];
                    // same-cell pairs are tested without minimum image, as the
                    // reference does (CellManager.cpp:246-262)
                    same = s_nc[t] == c ? (int)0x80000000 : 0;
                } else {
                    q = site_frac(a.pos4[j], box, LE, delta);
                    q.w = j;
                }
                s_m[f] = a.mol[q.w] | same;
                const int x0 = __shfl_sync(0xffffffffu, q.x, 0), y0 = __shfl_sync(0xffffffffu, q.y, 0),
                          z0 = __shfl_sync(0xffffffffu, q.z, 0);
                const int d[3] = {q.x - x0, q.y - y0, q.z - z0};
                const int at[3] = {x0 - s_c.x, y0 - s_c.y, z0 - s_c.z};
#pragma unroll
                for (int x = 0; x < 3; x++) {
                    const int lo = __reduce_min_sync(0xffffffffu, d[x]), hi = __reduce_max_sync(0xffffffffu, d[x]);
                    if (lane == 0) {
                        s_lo[x][ch] = (float)at[x] + (float)lo;
                        s_hi[x][ch] = (float)at[x] + (float)hi;
                    }
                }
                if (f >= cnt) q.w = -1;
                s_q[f] = q;
            }
            __syncthreads();
            if (i < 0) continue;
            const float hi = far ? 3.4e38f : (float)(a.rl2 * (1.0 + 1e-5)), lo = far ? -1.f : (float)(a.rl2 * (1.0 - 1e-5));
            // lane ch: how far chunk ch's box stays from the site (periodic;
            // under shear x is left out, its images slide)
            bool near = lane < nchunk;
            if (near) {
                auto gap = [&](int x, float di, float s) {
                    const float u = s_lo[x][lane] - di, v = s_hi[x][lane] - di;
                    // the box's nearest images: itself, one period down, one up
                    const float P = 4294967296.f;
                    auto away = [](float a, float b) { return fmaxf(fmaxf(a, -b), 0.f); };
                    return fminf(away(u, v), fminf(away(u - P, v - P), away(u + P, v + P))) * s;
                };
                const float gx = LE ? 0.f : gap(0, dix, sx), gy = gap(1, diy, sy), gz = gap(2, diz, sz);
                near = fmaf(gx, gx, fmaf(gy, gy, gz * gz)) < hi * 1.0001f;
            }
            for (unsigned todo = __ballot_sync(0xffffffffu, near); todo; todo &= todo - 1) {
                const int k = (__ffs(todo) - 1) * 32 + lane;
                const int4 q = s_q[k];
                const int ix = LE ? le_dx_frac(fi.x, fi.y, q.x, q.y, dfrac) : q.x - fi.x;
                const float dx = (float)ix * sx, dy = (float)(q.y - fi.y) * sy, dz = (float)(q.z - fi.z) * sz;
                const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
                bool take = r2 < lo;
                if (r2 < hi && !take && q.w >= 0) {
                    const bool pbc = s_m[k] >= 0;
                    take = ref_r2(a.pos4[i], a.pos4[q.w], box, pbc, LE && pbc, delta) < a.rl2;
                }
                take = take && q.w >= 0;
                const bool same = take && (a.mol_sites ? (unsigned)(q.w - mi * a.mol_sites) < (unsigned)a.mol_sites
                                                       : (s_m[k] & 0x7fffffff) == mi);
                if (same || (take && a.excl_intermol)) {   // the site itself is of its own molecule
                    take = q.w != i;
                    for (int e = e0; e < e1; e++)
                        if (a.excl[e] == q.w) { take = false; break; }
                }
                const unsigned m = __ballot_sync(0xffffffffu, take);
                if (take) {
                    const int at = count + __popc(m & ((1u << lane) - 1));
                    if (at < a.max_nbr) a.nbr[(size_t)at * a.n + i] = q.w | (same ? (int)0x80000000 : 0);
                }
                count += __popc(m);
            }
        }
        if (i >= 0 && lane == 0) {
            if (count > a.max_nbr) {
                atomicOr(a.status, ST_LIST_OVERFLOW);
                count = a.max_nbr;
            }
            a.nnbr[i] = count;
        }
    }
    // the block that finishes last counts the build and lowers the flag
    __syncthreads();
    if (threadIdx.x == 0 && atomicAdd(a.ticket, 1u) == gridDim.x - 1) {
        *a.ticket = 0;
        a.flags[5] = 0;
        a.flags[1] += 1;
        a.flags[0] = 0;
        if (LE) a.le[SC_LE_B - SC_LE] = *a.le;   // the offset this list was built for
    }
}

void launch_nlist(Ctx &c, bool force_rebuild) {
    if (force_rebuild) {
        int one = 1;
        cudaMemcpyAsync(c.flags, &one, sizeof(int), cudaMemcpyHostToDevice, c.stream);
        c.list_built = 1;
    }
    const Box *dbox = c.npt ? c.dbox : nullptr;
    double *le = c.ip.strain_rate != 0.0 && c.integrator_ready ? c.scal + SC_LE : nullptr;
    if (c.grid.use_cells)
        k_cells<<<CELL_CTAS, CELL_THREADS, 0, c.stream>>>(c.n, c.pos4, c.grid, c.box, le, c.pl.cell_of,
                                                          c.pl.cell_slot, c.pl.cell_count, c.pl.cell_start,
                                                          c.pl.cell_fill, c.pl.cell_q, c.pl.group, c.pl.ngroup,
                                                          c.flags, dbox);
    BuildArgs a;
    a.n = c.n; a.max_nbr = c.pl.max_nbr; a.pos4 = c.pos4; a.disp4 = c.disp4; a.mol = c.mol;
    a.excl_off = c.excl_off; a.excl = c.excl; a.excl_intermol = c.excl_intermol; a.mol_sites = c.mol_sites;
    a.cell_start = c.pl.cell_start; a.cell_q = c.pl.cell_q;
    a.group = c.grid.use_cells ? c.pl.group : nullptr;
    a.ngroup = c.pl.ngroup;
    a.g = c.grid; a.box = c.box;
    a.rl2 = c.pl.rl2; a.nbr = c.pl.nbr; a.nnbr = c.pl.nnbr; a.status = c.status; a.flags = c.flags;
    a.ticket = (unsigned *)(c.flags + 4);
    a.le = le;
    a.dbox = dbox;
    // blocks loop over the groups, so that a step without a rebuild launches
    // little more than the device holds at once (five a multiprocessor)
    const int groups = (c.n + NB_SITES - 1) / NB_SITES + c.grid.ncell, nb = groups < c.sms * 6 ? groups : c.sms * 6;
    if (a.le)
        k_build<true><<<nb, NB_SITES * 32, 0, c.stream>>>(a);
    else
        k_build<false><<<nb, NB_SITES * 32, 0, c.stream>>>(a);
}

}  // namespace smd
