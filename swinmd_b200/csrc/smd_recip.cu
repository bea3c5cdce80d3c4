// Ewald reciprocal-space sum for point charges (EwaldForce::set_up and
// EwaldForce::reciprocal_term, src/forces/EwaldForce.cpp:198-257, 529-698).
//
//   k set : n = (nx, ny, nz), half space (nx > 0, or nx = 0 and ny > 0, or
//           nx = ny = 0 and nz > 0), k = 2 pi n / L, k^2 < kCut^2
//   S(k)  = sum_i q_i exp(i k.r_i)                  (q: scaled charges)
//   E     = sum_k 4 pi/V exp(-k^2/4a^2)/k^2 |S(k)|^2
//   F_i  += k 8 pi/V exp(-k^2/4a^2)/k^2 (q_i sin(k.r_i) Re S - q_i cos(k.r_i) Im S)
//   W_ab += E_k (delta_ab - 2 (1/4a^2 + 1/k^2) k_a k_b)  (long virial)
//
// The passes go by columns of the k set, (nx, ny) with nz = -m .. m (nz =
// 1 .. m for nx = ny = 0).  Per site exp(i k.r) = A Z^nz with A = X^nx Y^ny,
// so a column's sums for +nz and -nz are four real products over the sites,
//   P = sum Re A Re Z^nz,  Q = sum Im A Im Z^nz,  R = sum Re A Im Z^nz,
//   T = sum Im A Re Z^nz:  S(+nz) = (P - Q, R + T),  S(-nz) = (P + Q, T - R),
// four FMAs for two k, and with g = 2c conj S the force takes, per column,
//   T0 = sum_nz (g+ + g-) Re Z^nz + i (g+ - g-) Im Z^nz   and the same with nz
// weights, eight FMAs for two k.  Everything is FP64 in both precision modes:
// one sine and cosine per site and axis and the powers of the factor replace
// one per (site, k), which bounded both passes (FP32 sincospif with FP64
// sums 57 + 73 us for 8000 ions and 2094 k; FP64 sincos 22 + 24 us for 2331
// sites and 900 k).
//
// Three kernels: partial sums over (column item x site chunk) blocks, a
// fixed-order reduction over chunks that also forms the force coefficients and
// the blocks' energies and virial, and a per-site force pass, one more block of
// which adds those up.
//
// Sheared cell (SLLOD with Lees-Edwards images; no reference code): the
// images of the box with offset d form the lattice a1 = (Lx, 0, 0),
// a2 = (d, Ly, 0), a3 = (0, 0, Lz), whose reciprocal vectors give
// k(n) = 2 pi (nx / Lx, (ny - nx t) / Ly, nz / Lz), t = d / Lx, with d
// reduced to [-Lx/2, Lx/2] (d and d + Lx are the same lattice).  The sums are
// those above over the half space of n with |k| < kcut for that lattice, so
// the columns change with d: k_le_columns rebuilds them on the device before
// every evaluation, in the order of the unsheared list, and the passes read
// the live count from the device.  The phase is n.(fractional coordinates):
// x's fraction becomes (x - d y / Ly) / Lx.
#include <cmath>
#include <vector>
#include <algorithm>
#include <cooperative_groups.h>
#include "smd_ctx.cuh"

namespace smd {

namespace cg = cooperative_groups;

constexpr double PI_R = 3.14159265358979323846;
constexpr int ES_THREADS = 128;   // column items per block of the sums pass
constexpr int ES_SITES = 32;      // sites per tile of the sums pass
constexpr int EF_THREADS = 64;    // sites per block of the force pass
constexpr int EF_COLS = 16;       // columns staged at a time in the force pass

struct EwArgs {
    int n, cap;           // sites; stride of the column arrays
    int nch;              // nz items per column
    int nX, nY, row;      // table entries per site: X^0.. [nX], Y^0.. [nY], Z^0.. [nch NZT]; the row's stride
    int tile;             // sites per tile of the sums pass
    const double4 *pos4;
    const double *tq;
    Box box;
    const double *le;     // Lees-Edwards offset on the device, or null
    const int4 *col;      // (nx, ny, largest nz, 0)
    const int *ncol;      // live columns
    double pi4V, aR4;
};

// the Lees-Edwards offset reduced to [-Lx/2, Lx/2]
__device__ __forceinline__ double le_reduced(const double *le, const Box &b) {
    const double d = le ? *le : 0.0;
    return d - b.L[0] * floor(d * b.inv[0] + 0.5);
}

// fractional coordinates along the (sheared) cell's vectors
__device__ __forceinline__ double3 ew_frac(const double4 &p, double dd, const Box &b) {
    const double fy = p.y * b.inv[1];
    return make_double3((p.x - dd * fy) * b.inv[0], fy, p.z * b.inv[2]);
}
// e^{2 pi i f}
__device__ __forceinline__ double2 ew_phase(double f) {
    double s, c;
    sincospi(2.0 * (f - rint(f)), &s, &c);
    return make_double2(c, s);
}
__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// The columns of the sheared cell (one block): candidates (nx, m) with nx in
// [0, nxm], m in [-nyr, nyr] and ny = m + rint(nx t) cover every n with
// |k| < kcut (|ny - nx t| <= kcut Ly / 2 pi and |nx t - rint(nx t)| <= 1/2).
// Each thread takes a contiguous run of candidates, counts its columns, and
// after a block-wide exclusive scan writes them in candidate order.
constexpr int LC_THREADS = 256;
__global__ void __launch_bounds__(LC_THREADS) k_le_columns(int nxm, int nyr, int nzm, Box box, const double *le,
                                                           double kc2, int4 *col, int *ncol_out, int *nk_out) {
    __shared__ int s_w[2][LC_THREADS / 32];
    const double PI2 = 6.283185307179586476925;
    const double t = le_reduced(le, box) * box.inv[0];
    const int nys = 2 * nyr + 1, total = (nxm + 1) * nys;
    const int per = (total + LC_THREADS - 1) / LC_THREADS;
    const int c0 = min(total, (int)threadIdx.x * per), c1 = min(total, c0 + per);
    // the column's largest nz, -1 for no member of the half space
    auto column = [&](int ci, int &nx, int &ny) {
        nx = ci / nys;
        ny = ci - nx * nys - nyr + (int)rint(nx * t);
        if (nx == 0 && ny < 0) return -1;
        const double kx = PI2 * nx * box.inv[0], ky = PI2 * (ny - nx * t) * box.inv[1];
        for (int nz = nzm; nz >= (nx == 0 && ny == 0 ? 1 : 0); nz--) {
            const double kz = PI2 * nz * box.inv[2];
            if (kx * kx + ky * ky + kz * kz < kc2) return nz;
        }
        return -1;
    };
    int cnt = 0, nk = 0;
    for (int ci = c0; ci < c1; ci++) {
        int nx, ny;
        const int m = column(ci, nx, ny);
        if (m >= 0) {
            cnt++;
            nk += nx == 0 && ny == 0 ? m : 2 * m + 1;
        }
    }
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int inc = cnt;
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += v;
    }
    nk = warp_sum(nk);
    if (lane == 31) { s_w[0][w] = inc; s_w[1][w] = nk; }
    __syncthreads();
    int before = 0, nall = 0, kall = 0;
    for (int q = 0; q < LC_THREADS / 32; q++) {
        if (q < w) before += s_w[0][q];
        nall += s_w[0][q];
        kall += s_w[1][q];
    }
    if (threadIdx.x == 0) { *ncol_out = nall; *nk_out = kall; }
    int at = before + inc - cnt;
    for (int ci = c0; ci < c1; ci++) {
        int nx, ny;
        const int m = column(ci, nx, ny);
        if (m >= 0) col[at++] = make_int4(nx, ny, m, 0);
    }
}

// Partial sums, part[chunk][nz][P Q R T][cap].  A thread owns NZT nz of one
// column (items ordered nz range by nz range, so that a warp's Z loads are
// broadcasts and its Y loads consecutive) and runs over the block's chunk of
// sites, whose factor powers stand in shared memory tile by tile.  The 4 NZT
// running sums in registers give 4 NZT FMAs per 2 + NZT shared loads.  8000
// ions, 2094 k: 13.8 us, of which FP64 issue would take 2 (34 M FMAs; pipe 27 %
// busy): waits for shared memory and the tiles' barriers with few warps a block.
template <int NZT>
__global__ void __launch_bounds__(ES_THREADS) k_ew_sums(EwArgs a, double *part) {
    extern __shared__ double2 s_tab[];   // [tile][row]
    const int ncol = *a.ncol, items = ncol * a.nch;
    const int it = blockIdx.x * ES_THREADS + threadIdx.x;
    if ((int)(blockIdx.x * ES_THREADS) >= items) return;   // block-uniform
    const int rng = it / ncol, ci = it - rng * ncol;
    int4 cc = make_int4(0, 0, -1, 0);
    if (it < items) cc = a.col[ci];
    const bool own = cc.z >= rng * NZT;
    const int ox = cc.x, oy = a.nX + abs(cc.y), oz = a.nX + a.nY + rng * NZT;
    const double ysg = cc.y < 0 ? -1.0 : 1.0;
    const int per = (a.n + gridDim.y - 1) / gridDim.y;
    const int s0 = blockIdx.y * per, s1 = min(a.n, s0 + per);
    const double dd = le_reduced(a.le, a.box);
    double P[NZT], Q[NZT], R[NZT], T[NZT];
#pragma unroll
    for (int j = 0; j < NZT; j++) P[j] = Q[j] = R[j] = T[j] = 0.0;
    for (int base = s0; base < s1; base += a.tile) {
        const int cnt = min(a.tile, s1 - base);
        __syncthreads();
        for (int e = threadIdx.x; e < 3 * cnt; e += ES_THREADS) {
            const int ax = e / cnt, q = e - ax * cnt;
            const double4 p = a.pos4[base + q];
            const double3 f = ew_frac(p, dd, a.box);
            const double2 z = ew_phase(ax == 0 ? f.x : (ax == 1 ? f.y : f.z));
            double2 *tp = s_tab + q * a.row + (ax == 0 ? 0 : (ax == 1 ? a.nX : a.nX + a.nY));
            const int len = ax == 0 ? a.nX : (ax == 1 ? a.nY : a.nch * NZT);
            double2 v = make_double2(ax == 0 ? a.tq[(int)p.w] : 1.0, 0.0);   // the charge rides on X
            for (int m = 0; m < len; m++) {
                tp[m] = v;
                v = cmul(v, z);
            }
        }
        __syncthreads();
        if (!own) continue;
        const double2 *tp = s_tab;
#pragma unroll 2
        for (int q = 0; q < cnt; q++, tp += a.row) {
            const double2 X = tp[ox], Y = tp[oy];
            const double yi = Y.y * ysg;
            const double ar = X.x * Y.x - X.y * yi, ai = X.x * yi + X.y * Y.x;
#pragma unroll
            for (int j = 0; j < NZT; j++) {
                const double2 Z = tp[oz + j];
                P[j] = fma(ar, Z.x, P[j]);
                Q[j] = fma(ai, Z.y, Q[j]);
                R[j] = fma(ar, Z.y, R[j]);
                T[j] = fma(ai, Z.x, T[j]);
            }
        }
    }
    if (!own) return;
#pragma unroll
    for (int j = 0; j < NZT; j++) {
        double *o = part + ((size_t)blockIdx.y * a.nch * NZT + rng * NZT + j) * 4 * a.cap + ci;
        o[0] = P[j];
        o[a.cap] = Q[j];
        o[2 * (size_t)a.cap] = R[j];
        o[3 * (size_t)a.cap] = T[j];
    }
}

// S(+-k) in fixed chunk order for 32 columns at one nz: energy and long virial
// (tot[nz][block of columns][8]: E, xx, yy, zz, xy, xz, yz, 0) and the force
// coefficients 2c (conj S+ + conj S-), 2c (conj S+ - conj S-) (zero for an nz
// the column does not hold)
constexpr int ER_ROWS = 8, ER_COLS = 32;
__global__ void __launch_bounds__(32 * ER_ROWS) k_ew_reduce(EwArgs a, int nzp, int nzt, int chunks, const double *part,
                                                            double4 *coef, double *tot) {
    __shared__ double s_p[ER_ROWS][4][32];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int ncol = *a.ncol, ci = blockIdx.x * ER_COLS + tx, nz = blockIdx.y;
    if ((int)blockIdx.x * ER_COLS >= ncol) return;   // block-uniform
    const int4 cc = ci < ncol ? a.col[ci] : make_int4(0, 0, -1, 0);
    const bool live = cc.z >= nz / nzt * nzt;   // the sums pass wrote this slot
    double v[4] = {0, 0, 0, 0};
    if (live)
        for (int ch = ty; ch < chunks; ch += ER_ROWS) {
            const double *o = part + ((size_t)ch * nzp + nz) * 4 * a.cap + ci;
#pragma unroll
            for (int s = 0; s < 4; s++) v[s] += o[s * (size_t)a.cap];
        }
#pragma unroll
    for (int s = 0; s < 4; s++) s_p[ty][s][tx] = v[s];
    __syncthreads();
    if (ty > 0) return;
#pragma unroll
    for (int s = 0; s < 4; s++) {
        v[s] = s_p[0][s][tx];
        for (int r = 1; r < ER_ROWS; r++) v[s] += s_p[r][s][tx];
    }
    const bool origin = cc.x == 0 && cc.y == 0;
    const bool plus = nz <= cc.z && !(origin && nz == 0), minus = plus && nz > 0 && !origin;
    double e = 0, w[6] = {0, 0, 0, 0, 0, 0};   // xx yy zz xy xz yz
    double4 co = make_double4(0, 0, 0, 0);
    if (plus) {
        const double t = le_reduced(a.le, a.box) * a.box.inv[0];
        const double kx = 2 * PI_R * cc.x * a.box.inv[0], ky = 2 * PI_R * (cc.y - cc.x * t) * a.box.inv[1],
                     kz = 2 * PI_R * nz * a.box.inv[2];
        const double k2 = kx * kx + ky * ky + kz * kz;
        const double c = a.pi4V * (exp(-k2 * a.aR4) / k2);
        const double cp = v[0] - v[1], sp = v[2] + v[3];
        const double cm = minus ? v[0] + v[1] : 0.0, sm = minus ? v[3] - v[2] : 0.0;
        const double ep = c * (cp * cp + sp * sp), em = c * (cm * cm + sm * sm);
        const double coeff = 2.0 * (a.aR4 + 1.0 / k2);
        e = ep + em;
        const double d = (ep - em) * coeff;
        w[0] = e - e * coeff * kx * kx;
        w[1] = e - e * coeff * ky * ky;
        w[2] = e - e * coeff * kz * kz;
        w[3] = -e * coeff * kx * ky;
        w[4] = -d * kx * kz;
        w[5] = -d * ky * kz;
        co = make_double4(2 * c * (cp + cm), -2 * c * (sp + sm), 2 * c * (cp - cm), -2 * c * (sp - sm));
    }
    if (ci < ncol) coef[(size_t)ci * nzp + nz] = co;
    e = warp_sum(e);
#pragma unroll
    for (int q = 0; q < 6; q++) w[q] = warp_sum(w[q]);
    if (tx < 8) {
        double x = tx == 0 ? e : 0.0;
#pragma unroll
        for (int q = 0; q < 6; q++)
            if (tx == q + 1) x = w[q];
        tot[8 * ((size_t)nz * gridDim.x + blockIdx.x) + tx] = x;
    }
}

// The energy and the long virial from the live blocks' totals (nb of gx per
// nz) in a fixed order, each rounded to fixed point once; one block
__device__ __forceinline__ void ew_totals(int nzp, int gx, int nb, const double *tot, long long *acc,
                                          double (*s)[8]) {
    const int q = threadIdx.x & 7, row = threadIdx.x >> 3;
    double x = 0;
#pragma unroll 8
    for (int b = row; b < nb * nzp; b += EF_THREADS / 8) x += tot[8 * ((size_t)(b / nb) * gx + b % nb) + q];
    s[row][q] = x;
    __syncthreads();
    if (threadIdx.x >= 7) return;
    for (int r = 1; r < EF_THREADS / 8; r++) x += s[r][q];
    const int slots[7][2] = {{ACC_E_LONG, -1},       {ACC_LVIR + 0, -1},       {ACC_LVIR + 4, -1},
                             {ACC_LVIR + 8, -1},     {ACC_LVIR + 1, ACC_LVIR + 3},
                             {ACC_LVIR + 2, ACC_LVIR + 6}, {ACC_LVIR + 5, ACC_LVIR + 7}};
    const unsigned long long fx = (unsigned long long)to_fix(x, ACC_SCALE);
    atomicAdd((unsigned long long *)&acc[slots[q][0]], fx);
    if (slots[q][1] >= 0) atomicAdd((unsigned long long *)&acc[slots[q][1]], fx);
}

// Per-site force.  The blocks of a cluster (along y) split the columns, so
// that a few thousand sites fill the device; their partial forces meet in
// shared memory over the cluster and enter the fixed-point sum once.  A thread
// keeps its site's Z^nz and nz Z^nz of one nz range in registers, so a column costs two broadcast shared loads and eight FMAs per
// nz; the column's X^nx Y^ny follows from the one before along ny.  8000 ions,
// 2094 k: 22.5 us, of which FP64 issue would take 4 (67 M FMAs; pipe 32 % busy):
// the dependent FP64 chains of a column and the barriers between groups.
template <int NZT>
__global__ void __launch_bounds__(EF_THREADS) k_ew_force(EwArgs a, const double4 *coef, long long *frc, const double *tot,
                                                         long long *acc) {
    __shared__ double4 s_co[EF_COLS * NZT];
    __shared__ int4 s_col[EF_COLS];
    __shared__ double s_f[3][EF_THREADS], s_tot[EF_THREADS / 8][8];
    const int i = blockIdx.x * EF_THREADS + threadIdx.x;
    const bool own = i < a.n;
    const double dd = le_reduced(a.le, a.box);
    const double4 p = own ? a.pos4[i] : make_double4(0, 0, 0, 0);
    const double3 f = ew_frac(p, dd, a.box);
    const double2 z1 = ew_phase(f.z), y1 = ew_phase(f.y);
    const int ncol = *a.ncol, nzp = a.nch * NZT;
    if (blockIdx.x == gridDim.x - 1) {   // past the sites; its whole cluster leaves here
        if (blockIdx.y == 0)
            ew_totals(nzp, (a.cap + ER_COLS - 1) / ER_COLS, (ncol + ER_COLS - 1) / ER_COLS, tot, acc, s_tot);
        return;
    }
    const int per = (ncol + gridDim.y - 1) / gridDim.y;
    const int c0 = blockIdx.y * per, c1 = min(ncol, c0 + per);
    double Fx = 0, Fy = 0, Fz = 0;
    double2 zc = make_double2(1.0, 0.0);
    for (int rng = 0; rng < a.nch; rng++) {
        double zr[NZT], zi[NZT], nr[NZT], ni[NZT];
#pragma unroll
        for (int j = 0; j < NZT; j++) {
            zr[j] = zc.x; zi[j] = zc.y;
            const double nz = rng * NZT + j;
            nr[j] = nz * zc.x; ni[j] = nz * zc.y;
            zc = cmul(zc, z1);
        }
        int pnx = -1, pny = 0;
        double2 xy = make_double2(0, 0);
        for (int g0 = c0; g0 < c1; g0 += EF_COLS) {
            const int cnt = min(EF_COLS, c1 - g0);
            __syncthreads();
            for (int e = threadIdx.x; e < cnt * NZT; e += EF_THREADS)
                s_co[e] = coef[(size_t)(g0 + e / NZT) * nzp + rng * NZT + e % NZT];
            if (threadIdx.x < cnt) s_col[threadIdx.x] = a.col[g0 + threadIdx.x];
            __syncthreads();
            for (int c = 0; c < cnt; c++) {
                const int4 cc = s_col[c];
                if (cc.x == pnx && cc.y == pny + 1) xy = cmul(xy, y1);
                else xy = ew_phase(cc.x * f.x + cc.y * f.y);
                pnx = cc.x;
                pny = cc.y;
                if (cc.z < rng * NZT) continue;
                double t0r = 0, t0i = 0, t1r = 0, t1i = 0;
#pragma unroll
                for (int j = 0; j < NZT; j++) {
                    const double4 g = s_co[c * NZT + j];
                    t0r = fma(g.x, zr[j], fma(-g.w, zi[j], t0r));
                    t0i = fma(g.y, zr[j], fma(g.z, zi[j], t0i));
                    t1r = fma(g.z, nr[j], fma(-g.y, ni[j], t1r));
                    t1i = fma(g.w, nr[j], fma(g.x, ni[j], t1i));
                }
                const double im0 = xy.x * t0i + xy.y * t0r;
                Fx = fma((double)cc.x, im0, Fx);
                Fy = fma((double)cc.y, im0, Fy);
                Fz += xy.x * t1i + xy.y * t1r;
            }
        }
    }
    s_f[0][threadIdx.x] = Fx; s_f[1][threadIdx.x] = Fy; s_f[2][threadIdx.x] = Fz;
    cg::cluster_group cl = cg::this_cluster();
    cl.sync();
    if (own && cl.block_rank() == 0) {
        for (int r = 1; r < (int)cl.num_blocks(); r++) {
            const double *o = cl.map_shared_rank(&s_f[0][0], r);
            Fx += o[threadIdx.x]; Fy += o[EF_THREADS + threadIdx.x]; Fz += o[2 * EF_THREADS + threadIdx.x];
        }
        const double q = a.tq[(int)p.w], t = dd * a.box.inv[0];
        frc[i] += to_fix(2 * PI_R * q * a.box.inv[0] * Fx, FRC_SCALE);
        frc[a.n + i] += to_fix(2 * PI_R * q * a.box.inv[1] * (Fy - t * Fx), FRC_SCALE);
        frc[2 * a.n + i] += to_fix(2 * PI_R * q * a.box.inv[2] * Fz, FRC_SCALE);
    }
    cl.sync();   // no block leaves while its shared memory may be read
}

// nz per item: the size in 5..8 that pads the longest column least
static int ew_nzt(int mmax) {
    int best = 8;
    for (int z = 7; z >= 5; z--)
        if ((mmax + z) / z * z < (mmax + best) / best * best) best = z;
    return best;
}

// the reduction's totals, behind the partial sums
static size_t ew_totals_size(const Recip &r) {
    return (size_t)8 * r.ew_nch * r.ew_nzt * ((r.ew_cap + ER_COLS - 1) / ER_COLS);
}

// the column buffers: ncap columns with |nx| <= nxm, |ny| <= nym, nz <= mmax
static int ew_alloc(Ctx &c, int ncap, int nxm, int nym, int mmax) {
    Recip &r = c.rc;
    auto realloc = [](auto **p, size_t cnt) -> bool {
        if (*p) cudaFree(*p);
        *p = nullptr;
        return cudaMalloc((void **)p, (cnt ? cnt : 1) * sizeof(**p)) == cudaSuccess;
    };
    r.ew_cap = ncap; r.ew_nx = nxm + 1; r.ew_ny = nym + 1;
    r.ew_nzt = ew_nzt(mmax);
    r.ew_nch = (mmax + r.ew_nzt) / r.ew_nzt;
    const int gx = (ncap * r.ew_nch + ES_THREADS - 1) / ES_THREADS;
    // site chunks: about two blocks of the sums pass per SM
    r.ew_chunks = std::max(1, std::min(c.sms, 2 * c.sms / std::max(gx, 1)));
    const size_t slots = (size_t)r.ew_nch * r.ew_nzt * ncap;
    if (!realloc(&r.ew_col, ncap) || !realloc(&r.ew_ncol, 1) || !realloc(&r.ew_coef, slots) ||
        !realloc(&r.ew_part, slots * 4 * r.ew_chunks + ew_totals_size(r)))
        return SMD_ERR_CUDA;
    return cudaMemset(r.ew_ncol, 0, sizeof(int)) == cudaSuccess ? 0 : SMD_ERR_CUDA;
}

// sheared cell: capacity for every candidate of k_le_columns
static int setup_recip_le(Ctx &c) {
    const double PI = PI_R;
    const double kCut = c.ew_kcut;
    c.rc.le_nx = (int)(kCut * c.box.L[0] / (2 * PI));
    c.rc.le_ny = (int)(kCut * c.box.L[1] / (2 * PI)) + 1;
    c.rc.le_nz = (int)(kCut * c.box.L[2] / (2 * PI));
    const long long cap = (long long)(c.rc.le_nx + 1) * (2 * c.rc.le_ny + 1);
    if (cap * (2 * c.rc.le_nz + 1) > (1 << 26)) return SMD_ERR_ARG;
    c.rc.nk = (int)(cap * (2 * c.rc.le_nz + 1));
    c.rc.nmax = std::max(c.rc.le_nx + c.rc.le_ny, c.rc.le_nz);
    if (c.rc.nk_dev) cudaFree(c.rc.nk_dev);
    c.rc.nk_dev = nullptr;
    if (cudaMalloc((void **)&c.rc.nk_dev, sizeof(int)) != cudaSuccess ||
        cudaMemset(c.rc.nk_dev, 0, sizeof(int)) != cudaSuccess)
        return SMD_ERR_CUDA;
    c.rc.le = 1;
    c.graph_dirty = 1;
    return ew_alloc(c, (int)cap, c.rc.le_nx, c.rc.le_ny + (c.rc.le_nx + 1) / 2, c.rc.le_nz);
}

int setup_recip(Ctx &c) {
    const double PI = 3.14159265358979323846;
    if (!(c.ewald_on || c.mp_on) || c.box.L[0] <= 0) return 0;
    // SLLOD shear with the point-charge sum: the k list follows the offset
    if (c.ewald_on && !c.mp_on && c.integrator_ready && c.ip.strain_rate != 0.0) return setup_recip_le(c);
    c.rc.le = 0;
    const double kCut = c.ew_kcut, kCut2 = kCut * kCut;
    const double alpha2 = c.ew_alpha * c.ew_alpha, alphaR4 = 1.0 / (4.0 * alpha2);
    const int nxMax = (int)(kCut * c.box.L[0] / (2 * PI));
    const int nyMax = (int)(kCut * c.box.L[1] / (2 * PI));
    const int nzMax = (int)(kCut * c.box.L[2] / (2 * PI));
    const double vx = 2.0 * PI / c.box.L[0], vy = 2.0 * PI / c.box.L[1], vz = 2.0 * PI / c.box.L[2];
    std::vector<int> nxs, nys, nzs;
    std::vector<double> kxs, kys, kzs, coef;
    const double vol = c.box.L[0] * c.box.L[1] * c.box.L[2];
    const double pi4Volumer = 4.0 * PI * (1.0 / vol);
    for (int nx = 0; nx <= nxMax; nx++) {
        double kx = nx * vx;
        for (int ny = (nx == 0 ? 0 : -nyMax); ny <= nyMax; ny++) {
            double ky = ny * vy;
            for (int nz = ((nx == 0 && ny == 0) ? 1 : -nzMax); nz <= nzMax; nz++) {
                double kz = nz * vz;
                double k2 = kx * kx + ky * ky + kz * kz;
                if (k2 < kCut2) {
                    nxs.push_back(nx); nys.push_back(ny); nzs.push_back(nz);
                    kxs.push_back(kx); kys.push_back(ky); kzs.push_back(kz);
                    coef.push_back(pi4Volumer * (exp(-k2 * alphaR4) / k2));
                }
            }
        }
    }
    const int nk = (int)nxs.size();
    c.rc.nk = nk;
    c.rc.nmax = 0;
    for (int k = 0; k < nk; k++)
        c.rc.nmax = std::max(c.rc.nmax, std::max(std::abs(nxs[k]), std::max(std::abs(nys[k]), std::abs(nzs[k]))));
    std::vector<int> kn(3 * (size_t)nk);
    std::vector<double> kv(3 * (size_t)nk);
    for (int k = 0; k < nk; k++) {
        kn[k] = nxs[k]; kn[nk + k] = nys[k]; kn[2 * nk + k] = nzs[k];
        kv[k] = kxs[k]; kv[nk + k] = kys[k]; kv[2 * nk + k] = kzs[k];
    }
    auto realloc = [](auto **p, size_t cnt) -> bool {
        if (*p) cudaFree(*p);
        *p = nullptr;
        return cudaMalloc((void **)p, (cnt ? cnt : 1) * sizeof(**p)) == cudaSuccess;
    };
    // the multipole passes' partial and total structure factors
    // partial sums, sums, block totals
    const size_t nsk = c.mp_on ? 6 * (size_t)nk * (MP_SK_CHUNKS + 1) + 8 * (size_t)((nk + MP_SK_BLOCK - 1) / MP_SK_BLOCK) : 0;
    if (!realloc(&c.rc.kn, 3 * (size_t)nk) || !realloc(&c.rc.kvec, 3 * (size_t)nk) ||
        !realloc(&c.rc.kcoef, (size_t)nk) || !realloc(&c.rc.sk, nsk))
        return SMD_ERR_CUDA;
    if (nk) {
        cudaMemcpy(c.rc.kn, kn.data(), kn.size() * sizeof(int), cudaMemcpyHostToDevice);
        cudaMemcpy(c.rc.kvec, kv.data(), kv.size() * sizeof(double), cudaMemcpyHostToDevice);
        cudaMemcpy(c.rc.kcoef, coef.data(), coef.size() * sizeof(double), cudaMemcpyHostToDevice);
    }
    c.graph_dirty = 1;
    if (c.ewald_on) {
        std::vector<int4> col;
        int mmax = 0;
        for (int k = 0; k < nk; k++) {
            if (k == 0 || nxs[k] != nxs[k - 1] || nys[k] != nys[k - 1]) col.push_back(make_int4(nxs[k], nys[k], 0, 0));
            col.back().z = std::max(col.back().z, nzs[k]);
            mmax = std::max(mmax, nzs[k]);
        }
        const int ncol = (int)col.size();
        const int r = ew_alloc(c, std::max(ncol, 1), nxMax, nyMax, mmax);
        if (r) return r;
        if (ncol && (cudaMemcpy(c.rc.ew_col, col.data(), ncol * sizeof(int4), cudaMemcpyHostToDevice) != cudaSuccess ||
                     cudaMemcpy(c.rc.ew_ncol, &ncol, sizeof(int), cudaMemcpyHostToDevice) != cudaSuccess))
            return SMD_ERR_CUDA;
    }
    return c.mp_on ? mp_recip_prepare(c) : 0;
}

// the live k count (the sheared cell's list is built on the device)
int recip_nk(Ctx &c, int *nk) {
    if (!c.rc.le) {
        *nk = c.rc.nk;
        return 0;
    }
    if (cudaStreamSynchronize(c.stream) != cudaSuccess) return SMD_ERR_CUDA;
    return cudaMemcpy(nk, c.rc.nk_dev, sizeof(int), cudaMemcpyDeviceToHost) == cudaSuccess ? 0 : SMD_ERR_CUDA;
}

template <int NZT>
static void launch_columns(Ctx &c, EwArgs a) {
    const Recip &r = c.rc;
    const int nzp = r.ew_nch * NZT, items = r.ew_cap * r.ew_nch;
    const int chunks = std::max(1, std::min(r.ew_chunks, (c.n + 7) / 8));
    const size_t smem = (size_t)a.tile * a.row * sizeof(double2);
    k_ew_sums<NZT><<<dim3((items + ES_THREADS - 1) / ES_THREADS, chunks), ES_THREADS, smem, c.stream>>>(a, r.ew_part);
    double *tot = r.ew_part + (size_t)nzp * r.ew_cap * 4 * r.ew_chunks;
    k_ew_reduce<<<dim3((r.ew_cap + ER_COLS - 1) / ER_COLS, nzp), ER_COLS * ER_ROWS, 0, c.stream>>>(
        a, nzp, NZT, chunks, r.ew_part, r.ew_coef, tot);
    // column ranges of the force pass (blocks of a cluster): at most eight
    // blocks a multiprocessor, at least four columns each
    const int nb = (c.n + EF_THREADS - 1) / EF_THREADS;
    int ranges = 8;
    while (ranges > 1 && (ranges * nb > c.sms * 8 || ranges * 4 > r.ew_cap)) ranges /= 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(nb + 1, ranges);   // the last column of blocks: the totals
    cfg.blockDim = dim3(EF_THREADS);
    cfg.stream = c.stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = ranges;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, k_ew_force<NZT>, a, (const double4 *)r.ew_coef, c.frc, (const double *)tot, c.acc);
}

void launch_recip(Ctx &c) {
    const Recip &r = c.rc;
    if (r.nk == 0) return;
    EwArgs a;
    a.n = c.n; a.cap = r.ew_cap; a.nch = r.ew_nch;
    a.nX = r.ew_nx; a.nY = r.ew_ny;
    a.row = (r.ew_nx + r.ew_ny + r.ew_nch * r.ew_nzt) | 1;   // odd: rows start in different banks
    a.tile = std::max(1, std::min(ES_SITES, (int)(48 * 1024 / (a.row * sizeof(double2)))));
    a.pos4 = c.pos4; a.tq = c.type_q; a.box = c.box;
    // sheared cell: the offset is the integrator's (zero before it starts)
    a.le = r.le && c.integrator_ready && c.ip.strain_rate != 0.0 ? c.scal + SC_LE : nullptr;
    a.col = r.ew_col; a.ncol = r.ew_ncol;
    const double vol = c.box.L[0] * c.box.L[1] * c.box.L[2];
    a.pi4V = 4.0 * PI_R * (1.0 / vol);
    a.aR4 = 1.0 / (4.0 * c.ew_alpha * c.ew_alpha);
    if (r.le)
        k_le_columns<<<1, LC_THREADS, 0, c.stream>>>(r.le_nx, r.le_ny, r.le_nz, c.box, a.le, c.ew_kcut * c.ew_kcut,
                                                     r.ew_col, r.ew_ncol, r.nk_dev);
    switch (r.ew_nzt) {
        case 5: launch_columns<5>(c, a); break;
        case 6: launch_columns<6>(c, a); break;
        case 7: launch_columns<7>(c, a); break;
        default: launch_columns<8>(c, a); break;
    }
}

}  // namespace smd
