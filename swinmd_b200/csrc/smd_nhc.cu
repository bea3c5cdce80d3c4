// Nose-Hoover chain velocity-Verlet integrator (NVT), optionally with SLLOD
// planar Couette shear and Lees-Edwards images.
//
// Chain: NHIntegrator::chain (src/integrators/NHIntegrator.cpp:1814-1912),
// 4 links, nc = 5 multiple steps, Suzuki-Yoshida weights (1/(2 - 2^(1/3)),
// 1 - 2 w, w), Q_0 = Nf kT tau^2, Q_k = kT tau^2 (:113-119).  With the
// barostat (smd_set_barostat: the reference's NpT run) the chain carries the
// isotropic MTK degree of freedom vlog with mass W = (Nf + 1) kT tau_P^2
// (:119): G_0 = 2 K + W vlog^2 - (Nf + 1) kT, G_log = (2 K (1 + 3/Nf) +
// 3 V (P_vir - P)) / W, and the velocity scale exp(-(v_1 + (1 + 3/Nf) vlog)
// dt/2); the drift is r' = r e^(2h) + v e^h S(h) dt with h = vlog dt/2 and
// S the sinh(h)/h series to h^8, and the box edges scale by e^(2h)
// (:390-419).  P_vir is the reference's -molVirt of the previous forces
// (:382, :635): the Lustig volume derivative of the pair energy,
// sum r du/dr / 3V, minus that of the tail correction (LJForce.cpp:136-250,
// 297-327), the trace of the pair virial here.  Without the barostat vlog
// stays 0 and the first link sees Nf kT: constant volume.
// Step order as NHIntegrator::run (:380-408, :628-644):
//   k_nhc_chain   chain half step on the kinetic energy of v (one thread),
//                 Lees-Edwards offset delta += g Ly dt, the list test limit
//   k_nhc_first   v *= s; [SLLOD v_x -= g dt/2 v_y]; v += dt/2 F/m; drift
//                 x += dt v_x + g dt (y + dt v_y / 2), y, z += dt v; wrap
//                 (y first, moving x by -/+ delta); displacement test
//   pair list (if flagged), forces at t + dt
//   k_nhc_second  v += dt/2 F/m; [SLLOD half step]; kinetic sums; the last
//                 block runs the second chain half step, the observables and
//                 the pressure tensors (peculiar velocities under shear)
//   k_nhc_scale   v *= s
// SLLOD (no reference code; Evans and Morriss, Statistical Mechanics of
// Nonequilibrium Liquids, ch. 6): v is the peculiar velocity, the streaming
// and the -g v_y e_x term are integrated exactly over their sub-steps.
// The pair list stays valid while 2 max|displacement| + |delta - delta_build|
// < skin: the displacement limit of each step is ((skin - |d delta|)/2)^2 and
// a rebuild is forced when that is not positive.
#include "smd_ctx.cuh"

namespace smd {

constexpr double KB_N = 0.0083145112;  // BOLTZMAN, src/NEMD_defs.h:108
constexpr int NHC_BLOCK = 128;

enum { Q_KE = 0, Q_AP = 1 /*6*/, Q_KEM = 7, Q_MP = 8 /*6*/, Q_MC = 14 /*9*/, NQ = 23 };

struct NhcArgs {
    int n, nmol, nblocks, mol_sites;
    const int *mol_off, *mol_atoms;
    double4 *pos4, *vel4, *disp4;
    int4 *fixq;
    int write_fixq;
    const long long *frc;
    long long *acc;
    double *scal, *partials;
    unsigned int *ticket, *status;
    int *flags;
    smd_observables *obs;
    double *series;
    int series_cap;
    double *avg;           // running sums of the observables (may be null)
    double *wrap;          // [3][nmol] box shifts applied to each molecule since the last upload
    Box box;
    double dt, kT, nf, tau, gamma, skin, volume;
    int atom_ndf, mol_ndf;
    double e_lrc, v_lrc, e_self;
    // barostat (npt): the box on the device, target pressure, W, the tail
    // correction's energy times volume, the smallest box scale the cell
    // grid covers and the box it was built for
    int npt;
    Box *dbox;
    double press, wbar, lrc_k, smin, L0[3];
};

// e^x of the chain's small arguments (velocities times a fraction of the time
// step): the Taylor series to x^8 below 1/64, where its remainder is under
// 2e-22, in two interleaved halves to shorten the dependent chain
__device__ __forceinline__ double chain_exp(double x) {
    if (!(fabs(x) < 0.015625)) return exp(x);
    const double y = x * x;
    const double even = 1.0 + y * (1.0 / 2 + y * (1.0 / 24 + y * (1.0 / 720 + y * (1.0 / 40320))));
    const double odd = 1.0 + y * (1.0 / 6 + y * (1.0 / 120 + y * (1.0 / 5040)));
    return fma(x, odd, even);
}

// one chain half step; returns the velocity scale (vnh in scal[SC_VNH..+3]);
// with the barostat also vlog, driven by the virial pressure pvir.  One
// thread's dependent chain: the way back up the links uses the exponentials
// of the way down (vnh[1..3] have not changed in between), the masses enter
// as reciprocals.  k_nhc_chain 15 -> 8 us, k_nhc_second 39 -> 15 us (4000 sites).
__device__ double chain_half(double (&vnh)[4], double ekin, const NhcArgs &a, double &vlog, double pvir, double vol) {
    const double q1 = a.kT * a.tau * a.tau, q0 = q1 * a.nf, iq1 = 1.0 / q1, iq0 = 1.0 / q0;
    const double w0 = 1.0 / (2.0 - cbrt(2.0));
    const int nc = 5;
    const double gkt = a.npt ? (a.nf + 1.0) * a.kT : a.nf * a.kT;
    const double odnf = 1.0 + 3.0 / a.nf, diff = pvir - a.press, iw = a.npt ? 1.0 / a.wbar : 0.0;
    double scale = 1.0;
    for (int i = 0; i < nc; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) {
            const double dts = (j == 1 ? 1.0 - 2.0 * w0 : w0) * a.dt / nc, dts2 = 0.5 * dts, dts4 = 0.25 * dts,
                         dts8 = 0.125 * dts;
            double g;
            vnh[3] += (q1 * vnh[2] * vnh[2] - a.kT) * iq1 * dts4;
            const double e3 = chain_exp(-vnh[3] * dts8);
            g = (q1 * vnh[1] * vnh[1] - a.kT) * iq1;
            vnh[2] = e3 * (vnh[2] * e3 + g * dts4);
            const double e2 = chain_exp(-vnh[2] * dts8);
            g = (q0 * vnh[0] * vnh[0] - a.kT) * iq1;
            vnh[1] = e2 * (vnh[1] * e2 + g * dts4);
            const double e1 = chain_exp(-vnh[1] * dts8);
            g = (2.0 * ekin + (a.npt ? a.wbar * vlog * vlog : 0.0) - gkt) * iq0;
            vnh[0] = e1 * (vnh[0] * e1 + g * dts4);
            double ex, e0 = 1.0;
            if (a.npt) {
                const double glog = (2.0 * ekin * odnf + 3.0 * vol * diff) * iw;
                e0 = chain_exp(-vnh[0] * dts8);
                vlog = e0 * (vlog * e0 + glog * dts4);
                ex = chain_exp(-(vnh[0] + vlog * odnf) * dts2);
            } else {
                ex = chain_exp(-vnh[0] * dts2);
            }
            scale *= ex;
            ekin = ekin * ex * ex;
            if (a.npt) {
                const double glog = (2.0 * ekin * odnf + 3.0 * vol * diff) * iw;
                vlog = e0 * (vlog * e0 + glog * dts4);
            }
            g = (2.0 * ekin + (a.npt ? a.wbar * vlog * vlog : 0.0) - gkt) * iq0;
            vnh[0] = e1 * (vnh[0] * e1 + g * dts4);
            g = (q0 * vnh[0] * vnh[0] - a.kT) * iq1;
            vnh[1] = e2 * (vnh[1] * e2 + g * dts4);
            g = (q1 * vnh[1] * vnh[1] - a.kT) * iq1;
            vnh[2] = e3 * (vnh[2] * e3 + g * dts4);
            vnh[3] += (q1 * vnh[2] * vnh[2] - a.kT) * iq1 * dts4;
        }
    return scale;
}

__global__ void k_nhc_chain(NhcArgs a) {
    if (threadIdx.x != 0) return;
    double vnh[4];
    for (int k = 0; k < 4; k++) vnh[k] = a.scal[SC_VNH + k];
    double vlog = a.scal[SC_VLOG];
    const double s = chain_half(vnh, a.scal[SC_EKIN], a, vlog, -a.scal[SC_MOLVIRT], a.scal[SC_VOL]);
    for (int k = 0; k < 4; k++) a.scal[SC_VNH + k] = vnh[k];
    a.scal[SC_SCALE] = s;
    if (a.npt) {
        // the drift's factors and the scaled box (NHIntegrator.cpp:390-419)
        a.scal[SC_VLOG] = vlog;
        const double term = 0.5 * a.dt * vlog, ex = exp(term), ex2 = ex * ex, arg2 = term * term;
        const double e2 = 1.0 / 6.0, e4 = e2 / 20.0, e6 = e4 / 42.0, e8 = e6 / 72.0;
        const double poly = ex * (1.0 + arg2 * (e2 + arg2 * (e4 + arg2 * (e6 + arg2 * e8)))) * a.dt;
        a.scal[SC_X2] = ex2;
        a.scal[SC_POLY] = poly;
        Box b = *a.dbox;
        bool small = false;
        for (int d = 0; d < 3; d++) {
            b.L[d] *= ex2;
            b.half[d] = 0.5 * b.L[d];
            b.inv[d] = 1.0 / b.L[d];
            small |= b.L[d] < a.smin * a.L0[d];
        }
        *a.dbox = b;
        a.scal[SC_VOL] = b.L[0] * b.L[1] * b.L[2];
        if (small) atomicOr(a.status, ST_BOX);
    }
    double lim = 0.5 * a.skin;
    if (a.gamma != 0.0) {
        const double Lx = a.box.L[0];
        double d = fmod(a.scal[SC_LE] + a.gamma * a.box.L[1] * a.dt, Lx);
        if (d < 0) d += Lx;
        a.scal[SC_LE] = d;
        double dd = fabs(d - a.scal[SC_LE_B]);
        dd = fmin(dd, Lx - dd);
        lim = 0.5 * (a.skin - dd);
        if (!(lim > 0)) {
            a.flags[0] = 1;
            lim = 0;
        }
    }
    a.scal[SC_DRMAX] = lim * lim;
}

__device__ __forceinline__ double3 nhc_force(const long long *frc, int n, int i) {
    return make_double3((double)frc[i] * FRC_INV, (double)frc[n + i] * FRC_INV, (double)frc[2 * n + i] * FRC_INV);
}

// one thread per molecule: scale, kick, drift, wrap, list test, box fractions
__global__ void __launch_bounds__(NHC_BLOCK) k_nhc_first(NhcArgs a) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    const double s = a.scal[SC_SCALE], delta = a.scal[SC_LE], drmax = a.scal[SC_DRMAX];
    const double hdt = 0.5 * a.dt, g = a.gamma;
    const Box bx = a.npt ? *a.dbox : a.box;
    const double x2 = a.npt ? a.scal[SC_X2] : 1.0, poly = a.npt ? a.scal[SC_POLY] : a.dt;
    bool rebuild = false, bad = false;
    if (m < a.nmol) {
        const int s0 = a.mol_sites ? m * a.mol_sites : a.mol_off[m], s1 = a.mol_sites ? s0 + a.mol_sites : a.mol_off[m + 1];
        double cx = 0, cy = 0, cz = 0, M = 0;
        for (int k = s0; k < s1; k++) {
            const int at = a.mol_sites ? k : a.mol_atoms[k];
            double4 v = a.vel4[at];   // w: 1/m
            const double3 f = nhc_force(a.frc, a.n, at);
            v.x *= s; v.y *= s; v.z *= s;
            if (g != 0.0) v.x -= g * hdt * v.y;
            v.x += hdt * v.w * f.x; v.y += hdt * v.w * f.y; v.z += hdt * v.w * f.z;
            double4 p = a.pos4[at];
            double drx, dry, drz;
            if (a.npt) {
                // r' = r e^(2h) + v e^h S(h) dt
                drx = (p.x * x2 + v.x * poly) - p.x;
                dry = (p.y * x2 + v.y * poly) - p.y;
                drz = (p.z * x2 + v.z * poly) - p.z;
                p.x = p.x * x2 + v.x * poly; p.y = p.y * x2 + v.y * poly; p.z = p.z * x2 + v.z * poly;
            } else {
                drx = a.dt * v.x + g * a.dt * (p.y + hdt * v.y);
                dry = a.dt * v.y; drz = a.dt * v.z;
                p.x += drx; p.y += dry; p.z += drz;
            }
            double4 d = a.disp4[at];
            d.x += drx; d.y += dry; d.z += drz;
            if (d.x * d.x + d.y * d.y + d.z * d.z > drmax) rebuild = true;
            if (!isfinite(p.x + p.y + p.z)) bad = true;
            a.vel4[at] = v;
            a.disp4[at] = d;
            a.pos4[at] = p;
            const double mass = 1.0 / v.w;
            cx += mass * p.x; cy += mass * p.y; cz += mass * p.z;
            M += mass;
        }
        cx /= M; cy /= M; cz /= M;
        // wrap the centre of mass: y first (Lees-Edwards), then x and z
        double wx = 0, wy = 0;
        if (cy >= bx.half[1]) { wy = -bx.L[1]; wx = -delta; }
        else if (cy < -bx.half[1]) { wy = bx.L[1]; wx = delta; }
        if (g == 0.0) wx = 0;
        wx = pbc1(cx + wx, bx.L[0], bx.half[0]) - cx;
        const double wz = pbc1(cz, bx.L[2], bx.half[2]) - cz;
        // the shifts so far, per molecule: Atom::realPos = position - shift
        if (a.wrap && (wx != 0.0 || wy != 0.0 || wz != 0.0)) {
            a.wrap[m] += wx;
            a.wrap[a.nmol + m] += wy;
            a.wrap[2 * a.nmol + m] += wz;
        }
        for (int k = s0; k < s1; k++) {
            const int at = a.mol_sites ? k : a.mol_atoms[k];
            double4 p = a.pos4[at];
            if (wx != 0.0 || wy != 0.0 || wz != 0.0) {
                p.x += wx; p.y += wy; p.z += wz;
                a.pos4[at] = p;
            }
            if (a.write_fixq) a.fixq[at] = site_frac(p, a.box, g != 0.0, delta);
        }
    }
    if (__any_sync(0xffffffffu, rebuild) && (threadIdx.x & 31) == 0) atomicOr(&a.flags[0], 1);
    if (bad) atomicOr(a.status, ST_NAN);
}

// one thread per molecule: second half kick, kinetic sums; last block:
// chain half step, observables, pressure tensors
__global__ void __launch_bounds__(NHC_BLOCK) k_nhc_second(NhcArgs a) {
    __shared__ double s_part[NHC_BLOCK / 32][NQ];
    __shared__ bool s_last;
    double part[NQ];
#pragma unroll
    for (int q = 0; q < NQ; q++) part[q] = 0.0;
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    const double hdt = 0.5 * a.dt, g = a.gamma;
    if (m < a.nmol) {
        const int s0 = a.mol_sites ? m * a.mol_sites : a.mol_off[m], s1 = a.mol_sites ? s0 + a.mol_sites : a.mol_off[m + 1];
        double px = 0, py = 0, pz = 0, cx = 0, cy = 0, cz = 0, M = 0;
        for (int k = s0; k < s1; k++) {
            const int at = a.mol_sites ? k : a.mol_atoms[k];
            double4 v = a.vel4[at];
            const double3 f = nhc_force(a.frc, a.n, at);
            v.x += hdt * v.w * f.x; v.y += hdt * v.w * f.y; v.z += hdt * v.w * f.z;
            if (g != 0.0) v.x -= g * hdt * v.y;
            a.vel4[at] = v;
            const double mass = 1.0 / v.w;
            const double mx = v.x * mass, my = v.y * mass, mz = v.z * mass;
            part[Q_KE] += (v.x * v.x + v.y * v.y + v.z * v.z) * mass;
            part[Q_AP + 0] += mx * v.x; part[Q_AP + 1] += mx * v.y; part[Q_AP + 2] += mx * v.z;
            part[Q_AP + 3] += my * v.y; part[Q_AP + 4] += my * v.z; part[Q_AP + 5] += mz * v.z;
            px += mx; py += my; pz += mz;
            const double4 p = a.pos4[at];
            cx += mass * p.x; cy += mass * p.y; cz += mass * p.z;
            M += mass;
        }
        cx /= M; cy /= M; cz /= M;
        part[Q_KEM] += (px * px + py * py + pz * pz) / M;
        part[Q_MP + 0] += px * px / M; part[Q_MP + 1] += px * py / M; part[Q_MP + 2] += px * pz / M;
        part[Q_MP + 3] += py * py / M; part[Q_MP + 4] += py * pz / M; part[Q_MP + 5] += pz * pz / M;
        for (int k = s0; k < s1; k++) {
            const int at = a.mol_sites ? k : a.mol_atoms[k];
            const double3 f = nhc_force(a.frc, a.n, at);
            const double4 p = a.pos4[at];
            const double rx = p.x - cx, ry = p.y - cy, rz = p.z - cz;
            part[Q_MC + 0] += f.x * rx; part[Q_MC + 1] += f.y * rx; part[Q_MC + 2] += f.z * rx;
            part[Q_MC + 3] += f.x * ry; part[Q_MC + 4] += f.y * ry; part[Q_MC + 5] += f.z * ry;
            part[Q_MC + 6] += f.x * rz; part[Q_MC + 7] += f.y * rz; part[Q_MC + 8] += f.z * rz;
        }
    }
    const int w = threadIdx.x >> 5;
    warp_sum_many<NQ>(part, s_part[w]);
    __syncthreads();
    if (threadIdx.x < NQ) {
        double v = 0;
        for (int q = 0; q < NHC_BLOCK / 32; q++) v += s_part[q][threadIdx.x];
        a.partials[(size_t)blockIdx.x * NQ + threadIdx.x] = v;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(a.ticket, 1u) == (unsigned)a.nblocks - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    // last block: totals in a fixed order (thread t sums the blocks t,
    // t + 128, ...), then the chain and the observables
    __shared__ StepTail S;
    __shared__ double tot[NQ];
    const double avg_old = tail_load(S, threadIdx.x, NHC_BLOCK, a.acc, a.avg, a.scal, a.obs, a.flags, a.status);
#pragma unroll
    for (int q = 0; q < NQ; q++) part[q] = 0.0;
    for (int b = threadIdx.x; b < a.nblocks; b += NHC_BLOCK)
#pragma unroll
        for (int q = 0; q < NQ; q++) part[q] += __ldcg(&a.partials[(size_t)b * NQ + q]);
    warp_sum_many<NQ>(part, s_part[w]);
    __syncthreads();
    if (threadIdx.x < NQ) {
        double v = 0;
        for (int q = 0; q < NHC_BLOCK / 32; q++) v += s_part[q][threadIdx.x];
        tot[threadIdx.x] = v;
    }
    __syncthreads();
    smd_observables &o = S.o;
    const double vol = a.npt ? S.scal[SC_VOL] : a.volume;
    // the tail correction of this volume (LJForce::long_range_correct,
    // recomputed every evaluation in NpT: E = K / V, virial -2 E, dU/dV = -2 E / V)
    const double e_lrc = a.npt ? a.lrc_k / vol : a.e_lrc;
    const double v_lrc = a.npt ? -2.0 * e_lrc : a.v_lrc;
    __shared__ double s_scale;
    if (threadIdx.x == 0) {
        double vnh[4];
        for (int k = 0; k < 4; k++) vnh[k] = S.scal[SC_VNH + k];
        double vlog = S.scal[SC_VLOG];
        const double s = chain_half(vnh, 0.5 * tot[Q_KE], a, vlog, -S.scal[SC_MOLVIRT], vol);
        for (int k = 0; k < 4; k++) a.scal[SC_VNH + k] = vnh[k];
        a.scal[SC_SCALE] = s;
        s_scale = s;
        if (a.npt) {
            a.scal[SC_VLOG] = vlog;
            // molVirt = -(sum r du/dr) / 3V + dU_lrc/dV (NHIntegrator.cpp:635)
            double tr = 0.0;
            for (int q = 0; q < 9; q += 4) tr += ((double)S.acc[ACC_VIR + q] + (double)S.acc[ACC_LVIR + q]) * ACC_INV;
            a.scal[SC_MOLVIRT] = -tr / (3.0 * vol) + v_lrc / vol;
        }
        o.zeta = vnh[0];
        const double s2 = s * s, keA = tot[Q_KE] * s2, keM = tot[Q_KEM] * s2;
        a.scal[SC_EKIN] = 0.5 * keA;
        o.ke_atom = 0.5 * keA;
        o.ke_mol = 0.5 * keM;
        o.t_atom = keA / (a.atom_ndf * KB_N);
        o.t_mol = keM / (a.mol_ndf * KB_N);
    } else if (threadIdx.x == 32) {
        double en[SMD_E_COUNT];
        acc_energies(S.acc, e_lrc, a.e_self, en);
        double ep = 0;
        for (int q = 0; q < SMD_E_COUNT; q++) {
            o.energy[q] = en[q];
            ep += en[q];
        }
        o.e_potential = ep;
        o.volume = vol;
        o.shear_offset = S.scal[SC_LE];
        o.step = S.step + 1;
        o.list_updates = S.list_updates;
        o.pairs_in_cutoff = S.acc[ACC_NPAIR] / 2;
        o.status = S.status;
        o.pad = 0;
    }
    __syncthreads();
    if (threadIdx.x < 9) {
        const int q = threadIdx.x;
        const int sym = q < 3 ? q : (q == 3 ? 1 : (q < 6 ? q - 1 : (q == 6 ? 2 : q - 3)));
        const double s2 = s_scale * s_scale;
        double vir = ((double)S.acc[ACC_VIR + q] + (double)S.acc[ACC_LVIR + q]) * ACC_INV;
        if (q == 0 || q == 4 || q == 8) vir -= v_lrc;
        o.mol_pressure[q] = (tot[Q_MP + sym] * s2 + vir - tot[Q_MC + q]) / vol;
        o.atom_pressure[q] = (tot[Q_AP + sym] * s2 + vir) / vol;
        o.virial[q] = vir;
    }
    __syncthreads();
    // the series' fifth value: xy, the shear stress under SLLOD
    tail_store(S, threadIdx.x, NHC_BLOCK, avg_old, a.acc, a.avg, a.obs, a.series, a.series_cap, o.atom_pressure[1],
               a.ticket);
}

__global__ void k_nhc_scale(int n, double4 *vel4, const double *scal) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double s = scal[SC_SCALE];
    double4 v = vel4[i];
    v.x *= s; v.y *= s; v.z *= s;
    vel4[i] = v;
}

// start: kinetic energy of the initial velocities, chain at rest, delta = 0
__global__ void k_nhc_start(int n, const double4 *vel4, double *scal, double skin, long long *acc) {
    __shared__ double s[256];
    double k = 0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const double4 v = vel4[i];
        k += (v.x * v.x + v.y * v.y + v.z * v.z) / v.w;
    }
    s[threadIdx.x] = k;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) s[threadIdx.x] += s[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        scal[SC_EKIN] = 0.5 * s[0];
        for (int q = 0; q < 4; q++) scal[SC_VNH + q] = 0.0;
        scal[SC_SCALE] = 1.0;
        scal[SC_LE] = 0.0;
        scal[SC_LE_B] = 0.0;
        scal[SC_DRMAX] = 0.25 * skin * skin;
    }
    __syncthreads();
    if (threadIdx.x < ACC_COUNT) acc[threadIdx.x] = 0;
}

namespace {
NhcArgs nhc_args(Ctx &c) {
    NhcArgs a;
    a.n = c.n; a.nmol = c.nmol; a.mol_sites = c.mol_sites;
    a.nblocks = (c.nmol + NHC_BLOCK - 1) / NHC_BLOCK;
    a.mol_off = c.mol_off; a.mol_atoms = c.mol_atoms;
    a.pos4 = c.pos4; a.vel4 = c.vel4; a.disp4 = c.disp4;
    a.fixq = c.fixq; a.write_fixq = c.precision == SMD_PREC_MIXED;
    a.frc = c.frc; a.acc = c.acc; a.scal = c.scal; a.partials = c.partials;
    a.ticket = c.ticket; a.status = c.status; a.flags = c.flags; a.obs = c.obs;
    a.series = c.series; a.series_cap = c.series_cap;
    a.avg = c.avg;
    a.wrap = c.wrap;
    a.box = c.box;
    a.dt = c.ip.timestep; a.kT = KB_N * c.ip.temperature; a.nf = c.ip.atom_ndf; a.tau = c.ip.coupl_const;
    a.gamma = c.ip.strain_rate; a.skin = c.cut_buffer;
    a.volume = c.box.L[0] * c.box.L[1] * c.box.L[2];
    a.atom_ndf = c.ip.atom_ndf; a.mol_ndf = c.ip.mol_ndf;
    a.e_lrc = c.e_lrc; a.v_lrc = c.v_lrc; a.e_self = c.e_self;
    a.npt = c.npt;
    a.dbox = c.dbox;
    a.press = c.npt_press;
    a.wbar = (c.ip.atom_ndf + 1.0) * a.kT * c.npt_tau * c.npt_tau;
    a.lrc_k = c.npt_lrc_k;
    a.smin = c.npt_smin;
    for (int d = 0; d < 3; d++) a.L0[d] = c.grid.L0[d];
    return a;
}
}  // namespace

void launch_nhc_first(Ctx &c) {
    NhcArgs a = nhc_args(c);
    k_nhc_chain<<<1, 32, 0, c.stream>>>(a);
    k_nhc_first<<<a.nblocks, NHC_BLOCK, 0, c.stream>>>(a);
}

void launch_nhc_second(Ctx &c) {
    NhcArgs a = nhc_args(c);
    k_nhc_second<<<a.nblocks, NHC_BLOCK, 0, c.stream>>>(a);
    k_nhc_scale<<<(c.n + 255) / 256, 256, 0, c.stream>>>(c.n, c.vel4, c.scal);
}

void launch_nhc_start(Ctx &c) {
    k_nhc_start<<<1, 256, 0, c.stream>>>(c.n, c.vel4, c.scal, c.cut_buffer, c.acc);
}

}  // namespace smd
