// Leap-frog Nose-Hoover integrator step (optionally with SHAKE), observables
// and thermostat update.
//
// One thread per molecule carries out, for the molecule's sites:
//  - unconstrained (LFIntegrator::run, src/integrators/LFIntegrator.cpp:
//    588-642): the implicit Nose-Hoover velocity iteration
//        v+ = v- + dt (F/m - zeta v),  v = (v+ + v-)/2   (to 1e-10, <= 10 passes)
//    then r += dt v+;
//  - SHAKE (LFIntegrator::shake, :1678-1827, NVT branch): v+ = v- + dt/m
//    (F - zeta P_mol/ns), unconstrained r' = r + dt v+, then the cyclic
//    3-distance SHAKE iteration in FP64 until every squared distance is
//    within 2 tol of its target (<= maxCount passes), v+ = (r' - r)/dt and
//    the SHAKE virial sum factor r'_ij (x) r_ij / dt^2;
// followed by the molecular centre of mass and momenta (:646-686), the
// pair-list displacement test (:307-315) and the molecule wrap into the box
// (:897-912).  The centre-of-mass drift removal the reference applies to v-
// at the start of the next step (:359-379) is applied here at the start of
// that step's update; forces do not depend on velocities, so the order is
// equivalent.  In the FP32 path the same thread also writes the sites' new
// 32-bit box fractions for the next step's pair kernel.
//
// Per-block partial sums (kinetic energies, kinetic pressure tensors, the
// molecular virial correction, sum m v-, the SHAKE virial) are combined by
// the last block to finish in a fixed order (deterministic); it then updates
// zeta (:688-722), temperatures, energies, the pressure tensors of
// Integrator::computePressure (src/Integrator.cpp:205-270, SHAKE virial added
// to the atomic tensor as at LFIntegrator.cpp:805-814) and clears the force
// accumulators for the next step.
#include <type_traits>
#include "smd_ctx.cuh"

namespace smd {

// scal[] layout
enum {
    SC_FNH = 0,     // zeta used by the next velocity update
    SC_FNHMI = 1,   // zeta(t - dt/2)
    SC_VOM = 2,     // 3: centre-of-mass velocity of v- to remove
    SC_APPLY = 5,   // nonzero: remove SC_VOM at the next update
    SC_COUNT = 8
};

// partial sums per block
enum {
    P_KEA = 0, P_KEM = 1, P_AP = 2 /*6*/, P_MP = 8 /*6*/, P_MC = 14 /*9*/, P_VM = 23 /*3*/,
    P_SV = 26 /*9*/, NPART = 35
};
constexpr int INT_BLOCK = 128;
constexpr double KB = 0.0083145112;  // BOLTZMAN, src/NEMD_defs.h:108

struct IntArgs {
    int n, nmol, nblocks, mol_sites;
    const int *mol_off, *mol_atoms;
    double4 *pos4, *vel4, *vtm4, *disp4;
    int4 *fixq;
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
    double dt, temperature, tau, drmax, total_mass, volume;
    int thermostat, atom_thermo, atom_ndf, mol_ndf, write_fixq;
    double e_lrc, v_lrc, e_self;
    const double *clen2;   // [nmol][3] squared constraint lengths
    double shake_tol;
    int shake_max;
};

__device__ __forceinline__ double3 fetch_force(const long long *frc, int n, int a) {
    return make_double3((double)frc[a] * FRC_INV, (double)frc[n + a] * FRC_INV,
                        (double)frc[2 * n + a] * FRC_INV);
}

__device__ __forceinline__ void pbc3(double &x, double &y, double &z, const Box &b) {
    x = pbc1(x, b.L[0], b.half[0]);
    y = pbc1(y, b.L[1], b.half[1]);
    z = pbc1(z, b.L[2], b.half[2]);
}

constexpr int MAX_MOL_SITES = 8;

// what the threads of a block found
struct IntFlags {
    bool nh_fail = false, rebuild = false, bad = false, shake_fail = false, shake_geom = false;
};

// the implicit Nose-Hoover velocity iteration of one site: v- in vm, v in v
// (in: the last on-step velocity), force f; returns v+
__device__ __forceinline__ double3 nose_hoover_site(const IntArgs &a, const double4 &vm, double4 &v, const double3 &f,
                                                    double fnh, IntFlags &F) {
    const double mr = v.w;
    double3 vp;
    if (a.thermostat == SMD_THERMO_NOSE_HOOVER) {
        double check2 = 1.0;   // |change of v|^2 of the last pass; to 1e-10
        int cnt = 0;
        while (check2 > 1e-20 && cnt < 11) {
            vp.x = vm.x + a.dt * (mr * f.x - fnh * v.x);
            vp.y = vm.y + a.dt * (mr * f.y - fnh * v.y);
            vp.z = vm.z + a.dt * (mr * f.z - fnh * v.z);
            const double nx = (vp.x + vm.x) * 0.5, ny = (vp.y + vm.y) * 0.5, nz = (vp.z + vm.z) * 0.5;
            const double ddx = nx - v.x, ddy = ny - v.y, ddz = nz - v.z;
            check2 = ddx * ddx + ddy * ddy + ddz * ddz;
            v.x = nx; v.y = ny; v.z = nz;
            cnt++;
        }
        if (cnt == 10) F.nh_fail = true;  // the reference's failure test
    } else {
        vp.x = vm.x + a.dt * mr * f.x;
        vp.y = vm.y + a.dt * mr * f.y;
        vp.z = vm.z + a.dt * mr * f.z;
    }
    return vp;
}

// the box shift that wraps a centre of mass, added to the molecule's count
__device__ __forceinline__ double3 wrap_shift(const IntArgs &a, int m, double cx, double cy, double cz) {
    const double3 w = make_double3(pbc1(cx, a.box.L[0], a.box.half[0]) - cx, pbc1(cy, a.box.L[1], a.box.half[1]) - cy,
                                   pbc1(cz, a.box.L[2], a.box.half[2]) - cz);
    // the shifts so far, per molecule: Atom::realPos = position - shift
    if (a.wrap && (w.x != 0.0 || w.y != 0.0 || w.z != 0.0)) {
        a.wrap[m] += w.x;
        a.wrap[a.nmol + m] += w.y;
        a.wrap[2 * a.nmol + m] += w.z;
    }
    return w;
}
__device__ __forceinline__ void put_position(const IntArgs &a, int at, double4 p, const double3 &w) {
    p.x += w.x; p.y += w.y; p.z += w.z;
    a.pos4[at] = p;
    if (a.write_fixq)
        a.fixq[at] = make_int4(frac32(p.x, a.box.inv[0]), frac32(p.y, a.box.inv[1]), frac32(p.z, a.box.inv[2]),
                               (int)p.w);
}

// One single-site molecule (ions, the Lennard-Jones fluid), site m: no
// indirection, every load issued before the arithmetic, the state written
// once.  Its molecular sums are the atomic ones and its virial correction
// vanishes (r = R), so 10 sums stand for the 35.
enum { P1_KE = 0, P1_AP = 1 /*6*/, P1_VM = 7 /*3*/, NPART1 = 10 };
__device__ __forceinline__ void integrate_site(const IntArgs &a, int m, double fnh, bool apply_vom, double vomx,
                                               double vomy, double vomz, double (&part)[NPART1], IntFlags &F) {
    double4 vm = a.vtm4[m], v = a.vel4[m], p = a.pos4[m], d = a.disp4[m];
    const double3 f = fetch_force(a.frc, a.n, m);
    if (apply_vom) {
        vm.x -= vomx; vm.y -= vomy; vm.z -= vomz;
        v.x -= vomx; v.y -= vomy; v.z -= vomz;
    }
    const double mass = vm.w;
    const double3 vp = nose_hoover_site(a, vm, v, f, fnh, F);
    const double drx = a.dt * vp.x, dry = a.dt * vp.y, drz = a.dt * vp.z;
    p.x += drx; p.y += dry; p.z += drz;
    d.x += drx; d.y += dry; d.z += drz;
    if (d.x * d.x + d.y * d.y + d.z * d.z > a.drmax) F.rebuild = true;
    v.x = (vp.x + vm.x) * 0.5; v.y = (vp.y + vm.y) * 0.5; v.z = (vp.z + vm.z) * 0.5;
    vm.x = vp.x; vm.y = vp.y; vm.z = vp.z;
    a.vel4[m] = v;
    a.vtm4[m] = vm;
    a.disp4[m] = d;
    if (!isfinite(p.x + p.y + p.z)) F.bad = true;
    const double mx = v.x * mass, my = v.y * mass, mz = v.z * mass;
    part[P1_KE] = (v.x * v.x + v.y * v.y + v.z * v.z) * mass;
    part[P1_AP + 0] = mx * v.x; part[P1_AP + 1] = mx * v.y; part[P1_AP + 2] = mx * v.z;
    part[P1_AP + 3] = my * v.y; part[P1_AP + 4] = my * v.z; part[P1_AP + 5] = mz * v.z;
    part[P1_VM + 0] = vm.x * mass; part[P1_VM + 1] = vm.y * mass; part[P1_VM + 2] = vm.z * mass;
    put_position(a, m, p, wrap_shift(a, m, p.x, p.y, p.z));
}

// One molecule's SHAKE step (LFIntegrator::shake, NVT branch) or, without
// constraints, site by site.  NS > 0 fixes the number of sites at compile
// time, so that every loop over sites and bonds unrolls and the sites' state
// stays in registers from one load to one store (three-site water); NS = 0
// takes the count at run time (up to MAX_MOL_SITES constrained sites, arrays
// in local memory).
template <int NS>
__device__ __forceinline__ void shake_mol(const IntArgs &a, int m, int s, int ns_rt, double fnh, bool apply_vom,
                                          double vomx, double vomy, double vomz, double (&part)[NPART], IntFlags &F) {
    constexpr int CAP = NS ? NS : MAX_MOL_SITES;
    const int ns = NS ? NS : ns_rt;
    int at[CAP];
    double4 p[CAP], vm[CAP], v[CAP], d[CAP];
    double3 f[CAP];
    double len2[3];
    for (int q = 0; q < ns; q++) at[q] = a.mol_sites ? s + q : a.mol_atoms[s + q];
    for (int q = 0; q < ns; q++) {
        vm[q] = a.vtm4[at[q]];   // w: mass
        v[q] = a.vel4[at[q]];    // w: 1/mass
        p[q] = a.pos4[at[q]];
        d[q] = a.disp4[at[q]];
        f[q] = fetch_force(a.frc, a.n, at[q]);
    }
    for (int q = 0; q < 3; q++) len2[q] = a.clen2[(size_t)m * 3 + q];
    // molecular momentum of the previous step (Molecule::momenta)
    double Px = 0, Py = 0, Pz = 0;
    for (int q = 0; q < ns; q++) {
        Px += v[q].x * vm[q].w; Py += v[q].y * vm[q].w; Pz += v[q].z * vm[q].w;
    }
    double rn[CAP][3], mr[CAP];
    for (int q = 0; q < ns; q++) {
        if (apply_vom) { vm[q].x -= vomx; vm[q].y -= vomy; vm[q].z -= vomz; }
        mr[q] = v[q].w;
        double vpx, vpy, vpz;
        if (a.thermostat == SMD_THERMO_NOSE_HOOVER) {
            vpx = vm[q].x + a.dt * mr[q] * (f[q].x - fnh * Px / ns);
            vpy = vm[q].y + a.dt * mr[q] * (f[q].y - fnh * Py / ns);
            vpz = vm[q].z + a.dt * mr[q] * (f[q].z - fnh * Pz / ns);
        } else {
            vpx = vm[q].x + a.dt * mr[q] * f[q].x;
            vpy = vm[q].y + a.dt * mr[q] * f[q].y;
            vpz = vm[q].z + a.dt * mr[q] * f[q].z;
        }
        rn[q][0] = p[q].x + a.dt * vpx; rn[q][1] = p[q].y + a.dt * vpy; rn[q][2] = p[q].z + a.dt * vpz;
    }
    const int nb = (ns == 3) ? 3 : ns - 1;
    const double tol2 = 2 * a.shake_tol;
    // the old bond vectors stay fixed during the iteration: their
    // minimum images once, and the SHAKE virial sum_k f_k n_k (x) o
    // as (sum_k f_k n_k) (x) o per bond at the end
    double ob[CAP][3], sfn[CAP][3];
    for (int i = 0; i < nb; i++) {
        const int nx = i + 1 == ns ? 0 : i + 1;
        double ox = p[i].x - p[nx].x, oy = p[i].y - p[nx].y, oz = p[i].z - p[nx].z;
        pbc3(ox, oy, oz, a.box);
        ob[i][0] = ox; ob[i][1] = oy; ob[i][2] = oz;
        sfn[i][0] = 0; sfn[i][1] = 0; sfn[i][2] = 0;
    }
    int count = 0;
    bool done = false;
    // Three sites: no branch on a bond that needs no correction (its factor is
    // 0; the warp's other molecules mostly need one) and, in place of a
    // division per correction, the factor's 1/B, B = 2 rr (m_i + m_j), kept
    // from the bond's last turn as y and brought up to date by 1/(1 - e) = (1 +
    // e)(1 + e^2)(1 + e^4) + O(e^8), e = 1 - B y.  Past |e| = 2^-7, where e^8
    // would show in FP64, y is divided out.  The sweeps are a serial chain of
    // about 90 corrections at a tolerance of 1e-8: 28.5 -> 22.9 us a step at
    // 777 and 2160 molecules.  In the bonds' own products (n_i.o_j updated in
    // place of positions) it took 24.3, with one lane per site 32.8 us.
    auto sweeps3 = [&](auto pbc) {
        double y[3] = {0, 0, 0};
        while (!done && count < a.shake_max) {
            done = true;
            bool geom = false;
#pragma unroll
            for (int i = 0; i < 3; i++) {
                const int nx = i == 2 ? 0 : i + 1;
                double nx_ = rn[i][0] - rn[nx][0], ny_ = rn[i][1] - rn[nx][1], nz_ = rn[i][2] - rn[nx][2];
                if (decltype(pbc)::value) pbc3(nx_, ny_, nz_, a.box);
                const double diff = len2[i] - (nx_ * nx_ + ny_ * ny_ + nz_ * nz_);
                const bool off = fabs(diff) > len2[i] * tol2;
                const double ox = ob[i][0], oy = ob[i][1], oz = ob[i][2];
                const double rr = ox * nx_ + oy * ny_ + oz * nz_;
                geom = geom || (off && rr < len2[i] * a.shake_tol);
                const bool need = off && !geom;   // from a failure on nothing moves
                done = done && !off;
                const double B = rr * (2 * (mr[i] + mr[nx]));
                double e = fma(-B, y[i], 1.0);
                if (need && !(fabs(e) <= 0x1p-7)) {
                    y[i] = 1.0 / B;
                    e = 0;
                }
                const double s = 1 + e, e2 = e * e, e4 = e2 * e2, q = y[i] * fma(s, e2, s);
                y[i] = fma(q, e4, q);
                const double factor = need ? diff * y[i] : 0.0, fi = factor * mr[i], fn = factor * mr[nx];
                sfn[i][0] += factor * nx_; sfn[i][1] += factor * ny_; sfn[i][2] += factor * nz_;
                rn[i][0] += fi * ox; rn[i][1] += fi * oy; rn[i][2] += fi * oz;
                rn[nx][0] -= fn * ox; rn[nx][1] -= fn * oy; rn[nx][2] -= fn * oz;
            }
            if (geom) { F.shake_geom = true; done = true; return; }
            count++;
        }
    };
    // the cyclic sweeps; PBC selects the minimum image of the new bond vectors
    auto sweeps = [&](auto pbc) {
        while (!done && count < a.shake_max) {
            done = true;
            for (int i = 0; i < nb; i++) {
                int nx = i + 1;
                if (nx == ns) nx = 0;
                double nx_ = rn[i][0] - rn[nx][0], ny_ = rn[i][1] - rn[nx][1], nz_ = rn[i][2] - rn[nx][2];
                if (decltype(pbc)::value) pbc3(nx_, ny_, nz_, a.box);
                const double r2 = nx_ * nx_ + ny_ * ny_ + nz_ * nz_;
                const double blen = len2[i < 3 ? i : 2];
                const double diff = blen - r2;
                if (fabs(diff) > blen * tol2) {
                    const double ox = ob[i][0], oy = ob[i][1], oz = ob[i][2];
                    const double rr = ox * nx_ + oy * ny_ + oz * nz_;
                    if (rr < blen * a.shake_tol) { F.shake_geom = true; done = true; count = a.shake_max; break; }
                    const double factor = diff / (2 * rr * (mr[i] + mr[nx]));
                    sfn[i][0] += factor * nx_; sfn[i][1] += factor * ny_; sfn[i][2] += factor * nz_;
                    rn[i][0] += factor * ox * mr[i]; rn[i][1] += factor * oy * mr[i]; rn[i][2] += factor * oz * mr[i];
                    rn[nx][0] -= factor * ox * mr[nx]; rn[nx][1] -= factor * oy * mr[nx];
                    rn[nx][2] -= factor * oz * mr[nx];
                    done = false;
                }
            }
            count++;
        }
    };
    // The minimum image leaves a bond vector unchanged while each component is
    // below half the box.  When every bond starts below a quarter of the box
    // the corrections (a small fraction of a bond length) cannot carry one
    // across half the box, so the sweeps skip the image test and give the
    // same numbers; a molecule split across the boundary takes the test.
    bool whole = true;
    for (int i = 0; i < nb; i++) {
        const int nx = i + 1 == ns ? 0 : i + 1;
        for (int c = 0; c < 3; c++) whole = whole && fabs(rn[i][c] - rn[nx][c]) < 0.5 * a.box.half[c];
    }
    auto run = [&](auto pbc) {
        if constexpr (NS == 3) sweeps3(pbc);
        else sweeps(pbc);
    };
    if (whole)
        run(std::integral_constant<bool, false>());
    else
        run(std::integral_constant<bool, true>());
    if (!done) F.shake_fail = true;
    for (int i = 0; i < nb; i++)
        for (int x = 0; x < 3; x++)
            for (int y = 0; y < 3; y++) part[P_SV + 3 * x + y] += sfn[i][x] * ob[i][y];
    double cx = 0, cy = 0, cz = 0, px = 0, py = 0, pz = 0, M = 0;
    for (int q = 0; q < ns; q++) {
        const double drx = rn[q][0] - p[q].x, dry = rn[q][1] - p[q].y, drz = rn[q][2] - p[q].z;
        p[q].x += drx; p[q].y += dry; p[q].z += drz;
        d[q].x += drx; d[q].y += dry; d[q].z += drz;
        if (d[q].x * d[q].x + d[q].y * d[q].y + d[q].z * d[q].z > a.drmax) F.rebuild = true;
        const double vpx = drx / a.dt, vpy = dry / a.dt, vpz = drz / a.dt;
        v[q].x = (vpx + vm[q].x) * 0.5; v[q].y = (vpy + vm[q].y) * 0.5; v[q].z = (vpz + vm[q].z) * 0.5;
        vm[q].x = vpx; vm[q].y = vpy; vm[q].z = vpz;
        a.vel4[at[q]] = v[q];
        a.vtm4[at[q]] = vm[q];
        a.disp4[at[q]] = d[q];
        if (!isfinite(p[q].x + p[q].y + p[q].z)) F.bad = true;
        const double mass = vm[q].w;
        const double mx = v[q].x * mass, my = v[q].y * mass, mz = v[q].z * mass;
        px += mx; py += my; pz += mz;
        cx += mass * p[q].x; cy += mass * p[q].y; cz += mass * p[q].z;
        M += mass;
        part[P_KEA] += (v[q].x * v[q].x + v[q].y * v[q].y + v[q].z * v[q].z) * mass;
        part[P_AP + 0] += mx * v[q].x; part[P_AP + 1] += mx * v[q].y; part[P_AP + 2] += mx * v[q].z;
        part[P_AP + 3] += my * v[q].y; part[P_AP + 4] += my * v[q].z; part[P_AP + 5] += mz * v[q].z;
        part[P_VM + 0] += vm[q].x * mass; part[P_VM + 1] += vm[q].y * mass; part[P_VM + 2] += vm[q].z * mass;
    }
    const double iM = 1.0 / M;
    cx *= iM; cy *= iM; cz *= iM;
    part[P_KEM] += (px * px + py * py + pz * pz) * iM;
    part[P_MP + 0] += px * px * iM; part[P_MP + 1] += px * py * iM; part[P_MP + 2] += px * pz * iM;
    part[P_MP + 3] += py * py * iM; part[P_MP + 4] += py * pz * iM; part[P_MP + 5] += pz * pz * iM;
    const double3 w = wrap_shift(a, m, cx, cy, cz);
    for (int q = 0; q < ns; q++) {
        // molecular virial correction sum_j f_j (r_j - R)  (Integrator.cpp:216-234)
        const double rx = p[q].x - cx, ry = p[q].y - cy, rz = p[q].z - cz;
        part[P_MC + 0] += f[q].x * rx; part[P_MC + 1] += f[q].y * rx; part[P_MC + 2] += f[q].z * rx;
        part[P_MC + 3] += f[q].x * ry; part[P_MC + 4] += f[q].y * ry; part[P_MC + 5] += f[q].z * ry;
        part[P_MC + 6] += f[q].x * rz; part[P_MC + 7] += f[q].y * rz; part[P_MC + 8] += f[q].z * rz;
        put_position(a, at[q], p[q], w);
    }
}

// A molecule without constraints, of any number of sites
__device__ __forceinline__ void free_mol(const IntArgs &a, int m, int s, int e, double fnh, bool apply_vom,
                                         double vomx, double vomy, double vomz, double (&part)[NPART], IntFlags &F) {
    double cx = 0, cy = 0, cz = 0, px = 0, py = 0, pz = 0, M = 0;
    for (int k = s; k < e; k++) {
        const int at = a.mol_atoms[k];
        double4 vm = a.vtm4[at];   // w: mass
        double4 v = a.vel4[at];    // w: 1/mass
        double4 p = a.pos4[at], d = a.disp4[at];
        const double3 f = fetch_force(a.frc, a.n, at);
        if (apply_vom) {
            vm.x -= vomx; vm.y -= vomy; vm.z -= vomz;
            v.x -= vomx; v.y -= vomy; v.z -= vomz;
        }
        const double mass = vm.w;
        const double3 vp = nose_hoover_site(a, vm, v, f, fnh, F);
        const double drx = a.dt * vp.x, dry = a.dt * vp.y, drz = a.dt * vp.z;
        p.x += drx; p.y += dry; p.z += drz;
        d.x += drx; d.y += dry; d.z += drz;
        if (d.x * d.x + d.y * d.y + d.z * d.z > a.drmax) F.rebuild = true;
        v.x = (vp.x + vm.x) * 0.5; v.y = (vp.y + vm.y) * 0.5; v.z = (vp.z + vm.z) * 0.5;
        vm.x = vp.x; vm.y = vp.y; vm.z = vp.z;
        a.vel4[at] = v;
        a.vtm4[at] = vm;
        a.disp4[at] = d;
        a.pos4[at] = p;
        if (!isfinite(p.x + p.y + p.z)) F.bad = true;
        const double mx = v.x * mass, my = v.y * mass, mz = v.z * mass;
        px += mx; py += my; pz += mz;
        cx += mass * p.x; cy += mass * p.y; cz += mass * p.z;
        M += mass;
        part[P_KEA] += (v.x * v.x + v.y * v.y + v.z * v.z) * mass;
        part[P_AP + 0] += mx * v.x; part[P_AP + 1] += mx * v.y; part[P_AP + 2] += mx * v.z;
        part[P_AP + 3] += my * v.y; part[P_AP + 4] += my * v.z; part[P_AP + 5] += mz * v.z;
        part[P_VM + 0] += vm.x * mass; part[P_VM + 1] += vm.y * mass; part[P_VM + 2] += vm.z * mass;
    }
    cx /= M; cy /= M; cz /= M;
    part[P_KEM] += (px * px + py * py + pz * pz) / M;
    part[P_MP + 0] += px * px / M; part[P_MP + 1] += px * py / M; part[P_MP + 2] += px * pz / M;
    part[P_MP + 3] += py * py / M; part[P_MP + 4] += py * pz / M; part[P_MP + 5] += pz * pz / M;
    const double3 w = wrap_shift(a, m, cx, cy, cz);
    for (int k = s; k < e; k++) {
        const int at = a.mol_atoms[k];
        const double3 f = fetch_force(a.frc, a.n, at);
        const double4 p = a.pos4[at];
        const double rx = p.x - cx, ry = p.y - cy, rz = p.z - cz;
        part[P_MC + 0] += f.x * rx; part[P_MC + 1] += f.y * rx; part[P_MC + 2] += f.z * rx;
        part[P_MC + 3] += f.x * ry; part[P_MC + 4] += f.y * ry; part[P_MC + 5] += f.z * ry;
        part[P_MC + 6] += f.x * rz; part[P_MC + 7] += f.y * rz; part[P_MC + 8] += f.z * rz;
        put_position(a, at, p, w);
    }
}

// KIND: single-site molecules, unconstrained molecules, SHAKE
enum IntKind { INT_SITES, INT_FREE, INT_SHAKE };

// What bounds it is latency: one molecule is one thread's dependent chain
// (loads, the SHAKE sweeps, stores), and the block that finishes last then
// forms the observables from every block's sums.  So each site's state is
// loaded at once and stored once, the 35 sums of a warp go through one
// transposed butterfly, and the finish reads and writes with many threads.
// Against one thread doing the finish and a reload per use: 20.8 -> 7 us at
// 500 sites, 40 -> 13 us at 62 500 sites, 47 -> 23 us with SHAKE at 2160
// molecules.
template <int KIND>
__global__ void __launch_bounds__(INT_BLOCK) k_integrate(IntArgs a) {
    constexpr int NP = KIND == INT_SITES ? (int)NPART1 : (int)NPART, NW = INT_BLOCK / 32;
    __shared__ double s_part[NW][NP];
    __shared__ bool s_last;
    double part[NP];
#pragma unroll
    for (int q = 0; q < NP; q++) part[q] = 0.0;

    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    const double fnh = a.scal[SC_FNH];
    const bool apply_vom = a.scal[SC_APPLY] != 0.0;
    const double vomx = a.scal[SC_VOM], vomy = a.scal[SC_VOM + 1], vomz = a.scal[SC_VOM + 2];
    IntFlags F;
    if (m < a.nmol) {
        if constexpr (KIND == INT_SITES) {
            integrate_site(a, m, fnh, apply_vom, vomx, vomy, vomz, part, F);
        } else {
            const int s = a.mol_sites ? m * a.mol_sites : a.mol_off[m];
            const int e = a.mol_sites ? s + a.mol_sites : a.mol_off[m + 1];
            const int ns = e - s;
            if (KIND == INT_SHAKE && ns == 3)
                shake_mol<3>(a, m, s, ns, fnh, apply_vom, vomx, vomy, vomz, part, F);
            else if (KIND == INT_SHAKE && ns > 1 && ns <= MAX_MOL_SITES)
                shake_mol<0>(a, m, s, ns, fnh, apply_vom, vomx, vomy, vomz, part, F);
            else
                free_mol(a, m, s, e, fnh, apply_vom, vomx, vomy, vomz, part, F);
        }
    }
    if (__any_sync(0xffffffffu, F.rebuild) && (threadIdx.x & 31) == 0) atomicOr(&a.flags[0], 1);
    if (F.nh_fail) atomicOr(a.status, ST_NH_ITER);
    if (F.bad) atomicOr(a.status, ST_NAN);
    if (F.shake_fail) atomicOr(a.status, ST_SHAKE_ITER);
    if (F.shake_geom) atomicOr(a.status, ST_SHAKE_GEOM);

    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    warp_sum_many<NP>(part, s_part[w]);
    __syncthreads();
    if (threadIdx.x < NP) {
        double v = 0;
        for (int q = 0; q < NW; q++) v += s_part[q][threadIdx.x];
        a.partials[(size_t)blockIdx.x * NP + threadIdx.x] = v;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned int t = atomicAdd(a.ticket, 1u);
        s_last = (t == (unsigned)a.nblocks - 1);
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();

    // ---- last block: totals in a fixed order ---------------------------
    // thread t sums the blocks t, t + 128, ... (every slot at once), then the
    // warps and the block as above (same order on every run)
    __shared__ StepTail S;
    __shared__ double tot[NPART];
    const double avg_old = tail_load(S, threadIdx.x, INT_BLOCK, a.acc, a.avg, a.scal, a.obs, a.flags, a.status);
#pragma unroll
    for (int q = 0; q < NP; q++) part[q] = 0.0;
    for (int b = threadIdx.x; b < a.nblocks; b += INT_BLOCK)
#pragma unroll
        for (int q = 0; q < NP; q++) part[q] += __ldcg(&a.partials[(size_t)b * NP + q]);
    warp_sum_many<NP>(part, s_part[w]);
    __syncthreads();
    if (threadIdx.x < NPART) {
        // single-site molecules: the molecular sums are the atomic ones, the
        // virial correction and SHAKE sums vanish
        const int t = threadIdx.x;
        const int src = KIND != INT_SITES                      ? t
                        : t == P_KEA || t == P_KEM             ? (int)P1_KE
                        : t >= P_AP && t < P_AP + 6            ? P1_AP + t - P_AP
                        : t >= P_MP && t < P_MP + 6            ? P1_AP + t - P_MP
                        : t >= P_VM && t < P_VM + 3            ? P1_VM + t - P_VM
                                                               : -1;
        double v = 0;
        if (src >= 0)
            for (int q = 0; q < NW; q++) v += s_part[q][src];
        tot[t] = v;
    }
    __syncthreads();
    smd_observables &o = S.o;
    if (w == 0 && lane < 9) {
        // virial and pressure tensors (Integrator::computePressure; SHAKE
        // virial added afterwards to the atomic tensor, LFIntegrator.cpp:805-814)
        const int q = lane;
        const int sym = q < 3 ? q : (q == 3 ? 1 : (q < 6 ? q - 1 : (q == 6 ? 2 : q - 3)));
        const double iV = 1.0 / a.volume;
        double vir = ((double)S.acc[ACC_VIR + q] + (double)S.acc[ACC_LVIR + q]) * ACC_INV;
        if (q == 0 || q == 4 || q == 8) vir -= a.v_lrc;
        o.mol_pressure[q] = (tot[P_MP + sym] + vir - tot[P_MC + q]) * iV;
        o.atom_pressure[q] = (tot[P_AP + sym] + vir) * iV;
        if (KIND == INT_SHAKE) {
            const double sv = tot[P_SV + q] / (a.dt * a.dt);
            vir += sv;
            o.atom_pressure[q] += sv * iV;
        }
        o.virial[q] = vir;
    } else if (w == 1 && lane == 0) {
        double en[SMD_E_COUNT];
        acc_energies(S.acc, a.e_lrc, a.e_self, en);
        double ep = 0;
        for (int q = 0; q < SMD_E_COUNT; q++) {
            o.energy[q] = en[q];
            ep += en[q];
        }
        o.e_potential = ep;
        o.volume = a.volume;
        o.step = S.step + 1;
        o.list_updates = S.list_updates;
        o.pairs_in_cutoff = S.acc[ACC_NPAIR] / 2;
        o.status = S.status;
        o.pad = 0;
        o.shear_offset = 0.0;
    } else if (w == 2 && lane == 0) {
        const double keA = tot[P_KEA], keM = tot[P_KEM];
        // Nose-Hoover zeta update (LFIntegrator.cpp:688-722)
        double zeta = 0.0;
        if (a.thermostat == SMD_THERMO_NOSE_HOOVER) {
            const double ndf = a.atom_thermo ? a.atom_ndf : a.mol_ndf;
            const double qq = ndf * KB * a.temperature * a.tau * a.tau;
            const double invqq = 1.0 / qq;
            const double ke = a.atom_thermo ? keA : keM, fnhmi = S.scal[SC_FNHMI];
            const double fnhpl = fnhmi + a.dt * invqq * (ke - ndf * KB * a.temperature);
            zeta = 0.5 * (fnhpl + fnhmi);
            a.scal[SC_FNHMI] = fnhpl;
        }
        a.scal[SC_FNH] = zeta;
        o.zeta = zeta;
        o.ke_atom = 0.5 * keA;
        o.ke_mol = 0.5 * keM;
        o.t_atom = keA / (a.atom_ndf * KB);
        o.t_mol = keM / (a.mol_ndf * KB);
    } else if (w == 3 && lane == 0) {
        // centre-of-mass drift of v- for the next step (LFIntegrator.cpp:359-379)
        const double vx = tot[P_VM] / a.total_mass, vy = tot[P_VM + 1] / a.total_mass,
                     vz = tot[P_VM + 2] / a.total_mass;
        a.scal[SC_VOM] = vx; a.scal[SC_VOM + 1] = vy; a.scal[SC_VOM + 2] = vz;
        a.scal[SC_APPLY] = (fabs(vx) > 1e-11 || fabs(vy) > 1e-11 || fabs(vz) > 1e-11) ? 1.0 : 0.0;
    }
    __syncthreads();
    tail_store(S, threadIdx.x, INT_BLOCK, avg_old, a.acc, a.avg, a.obs, a.series, a.series_cap,
               (o.atom_pressure[0] + o.atom_pressure[4] + o.atom_pressure[8]) / 3.0, a.ticket);
}

// State crosses the bus as the caller's [n][3] arrays, through c.stage; these
// put the fourth components (type, 1/m, m) in or leave them out.  Packing on the
// host cost a pass and freshly mapped pages per array: 62 500 sites up and down
// (and the launches of a segment around them) 2.4 -> 1.2 ms.
//
// keep: each site's minimum-image displacement adds to its displacement since
// the last list rebuild, and the rebuild flag is raised past half the skin;
// otherwise the next step rebuilds the list.
__global__ void k_put_positions(int n, const double *src, const int *type, double4 *pos4, double4 *disp4, Box b,
                                double drmax, int *flags, bool keep) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double4 p = make_double4(src[3 * (size_t)i], src[3 * (size_t)i + 1], src[3 * (size_t)i + 2], (double)type[i]);
    double4 d = make_double4(0, 0, 0, 0);
    if (keep) {
        const double4 o = pos4[i];
        d = disp4[i];
        d.x += pbc1(p.x - o.x, b.L[0], b.half[0]);
        d.y += pbc1(p.y - o.y, b.L[1], b.half[1]);
        d.z += pbc1(p.z - o.z, b.L[2], b.half[2]);
        if (d.x * d.x + d.y * d.y + d.z * d.z > drmax) atomicOr(&flags[0], 1);
    } else if (i == 0) {
        flags[0] = 1;
    }
    disp4[i] = d;
    pos4[i] = p;
}
__global__ void k_put_velocities(int n, const double *vel, const double *vtm, const double *mass, double4 *vel4,
                                 double4 *vtm4) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const size_t q = 3 * (size_t)i;
    vel4[i] = make_double4(vel[q], vel[q + 1], vel[q + 2], 1.0 / mass[i]);
    vtm4[i] = make_double4(vtm[q], vtm[q + 1], vtm[q + 2], mass[i]);
}
__global__ void k_get_state(int n, const double4 *pos4, const double4 *vel4, const double4 *vtm4, double *out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double4 *src[3] = {pos4, vel4, vtm4};
#pragma unroll
    for (int a = 0; a < 3; a++) {
        if (!src[a]) continue;
        const double4 v = src[a][i];
        double *o = out + 3 * ((size_t)a * n + i);
        o[0] = v.x; o[1] = v.y; o[2] = v.z;
    }
}

void launch_put_positions(Ctx &c, bool keep_list) {
    k_put_positions<<<(c.n + 255) / 256, 256, 0, c.stream>>>(c.n, c.stage, c.type, c.pos4, c.disp4, c.box, c.pl.drmax,
                                                             c.flags, keep_list);
}
void launch_put_velocities(Ctx &c, bool own_vtm) {
    const double *vel = c.stage + 3 * (size_t)c.n;
    k_put_velocities<<<(c.n + 255) / 256, 256, 0, c.stream>>>(c.n, vel, own_vtm ? vel + 3 * (size_t)c.n : vel, c.mass,
                                                              c.vel4, c.vtm4);
}
void launch_get_state(Ctx &c, bool pos, bool vel, bool vtm) {
    k_get_state<<<(c.n + 255) / 256, 256, 0, c.stream>>>(c.n, pos ? c.pos4 : nullptr, vel ? c.vel4 : nullptr,
                                                         vtm ? c.vtm4 : nullptr, c.stage);
}

void launch_integrate(Ctx &c) {
    IntArgs a;
    a.n = c.n; a.nmol = c.nmol; a.mol_sites = c.mol_sites;
    a.nblocks = (c.nmol + INT_BLOCK - 1) / INT_BLOCK;
    a.mol_off = c.mol_off; a.mol_atoms = c.mol_atoms;
    a.pos4 = c.pos4; a.vel4 = c.vel4; a.vtm4 = c.vtm4; a.disp4 = c.disp4;
    a.fixq = c.fixq; a.write_fixq = c.precision == SMD_PREC_MIXED;
    a.frc = c.frc; a.acc = c.acc; a.scal = c.scal; a.partials = c.partials;
    a.ticket = c.ticket; a.status = c.status; a.flags = c.flags; a.obs = c.obs;
    a.series = c.series; a.series_cap = c.series_cap;
    a.avg = c.avg;
    a.wrap = c.wrap;
    a.box = c.box;
    a.dt = c.ip.timestep; a.temperature = c.ip.temperature; a.tau = c.ip.coupl_const;
    a.drmax = c.pl.drmax; a.total_mass = c.total_mass;
    a.volume = c.box.L[0] * c.box.L[1] * c.box.L[2];
    a.thermostat = c.ip.thermostat; a.atom_thermo = c.ip.atom_thermo;
    a.atom_ndf = c.ip.atom_ndf; a.mol_ndf = c.ip.mol_ndf;
    a.e_lrc = c.e_lrc; a.v_lrc = c.v_lrc; a.e_self = c.e_self;
    a.clen2 = c.clen2; a.shake_tol = c.ip.shake_tol; a.shake_max = c.ip.shake_max_iter;
    if (c.ip.constraint == 2)
        k_integrate<INT_SHAKE><<<a.nblocks, INT_BLOCK, 0, c.stream>>>(a);
    else if (c.mol_sites == 1)
        k_integrate<INT_SITES><<<a.nblocks, INT_BLOCK, 0, c.stream>>>(a);
    else
        k_integrate<INT_FREE><<<a.nblocks, INT_BLOCK, 0, c.stream>>>(a);
}

// LFIntegrator::start (LFIntegrator.cpp:1172-1173): vtMinus = v - dt/2 F/m.
__global__ void k_start(int n, double dt, const long long *frc, const double4 *vel4,
                        double4 *vtm4) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double4 v = vel4[i];
    double4 vm = vtm4[i];
    const double3 f = fetch_force(frc, n, i);
    vm.x = v.x - 0.5 * dt * v.w * f.x;
    vm.y = v.y - 0.5 * dt * v.w * f.y;
    vm.z = v.z - 0.5 * dt * v.w * f.z;
    vtm4[i] = vm;
}

// Centre-of-mass velocity of v- for the first step, one block, fixed order.
__global__ void __launch_bounds__(1024) k_vom(int n, const double4 *vtm4, double total_mass, double *scal,
                      long long *acc) {
    __shared__ double s[32][3];
    double x = 0, y = 0, z = 0;
    // four loads of a thread in flight: 72 -> 20 us at 62 500 sites (256
    // threads, one load)
#pragma unroll 4
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        double4 v = vtm4[i];
        x += v.x * v.w; y += v.y * v.w; z += v.z * v.w;
    }
    x = warp_sum(x); y = warp_sum(y); z = warp_sum(z);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) { s[w][0] = x; s[w][1] = y; s[w][2] = z; }
    __syncthreads();
    if (w == 0) {
        x = warp_sum(s[lane][0]); y = warp_sum(s[lane][1]); z = warp_sum(s[lane][2]);
    }
    if (threadIdx.x == 0) {
        const double vx = x / total_mass, vy = y / total_mass, vz = z / total_mass;
        scal[SC_VOM] = vx; scal[SC_VOM + 1] = vy; scal[SC_VOM + 2] = vz;
        scal[SC_APPLY] = (fabs(vx) > 1e-11 || fabs(vy) > 1e-11 || fabs(vz) > 1e-11) ? 1.0 : 0.0;
        scal[SC_FNH] = 0.0;
        scal[SC_FNHMI] = 0.0;
    }
    __syncthreads();
    if (threadIdx.x < ACC_COUNT) acc[threadIdx.x] = 0;
}

void launch_start_velocities(Ctx &c) {
    k_start<<<(c.n + 255) / 256, 256, 0, c.stream>>>(c.n, c.ip.timestep, c.frc, c.vel4, c.vtm4);
    k_vom<<<1, 1024, 0, c.stream>>>(c.n, c.vtm4, c.total_mass, c.scal, c.acc);
}

// Fixed-point forces to the reference's per-atom FP64 Vector3 layout.
__global__ void k_forces_out(int n, const long long *frc, double *out) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    out[3 * i] = (double)frc[i] * FRC_INV;
    out[3 * i + 1] = (double)frc[n + i] * FRC_INV;
    out[3 * i + 2] = (double)frc[2 * n + i] * FRC_INV;
}

void launch_finalize_forces(Ctx &c, double *f_out_dev) {
    k_forces_out<<<(c.n + 255) / 256, 256, 0, c.stream>>>(c.n, c.frc, f_out_dev);
}

// EwaldForce::intraMolCorrect (src/forces/EwaldForce.cpp:709-813): for
// every excluded site pair inside a molecule, -q_i q_j erf(a r)/r into the
// energy; with no constraints also the force q_i q_j (erf(a r)/r -
// 2a/sqrt(pi) exp(-a^2 r^2))/r^2 r_ij on i (and its negative on j), which
// the reference leaves out of the virial.  One thread per molecule owns its
// sites' forces.
__global__ void k_intra_ewald(int nmol, int n, const int *mol_off, const int *mol_atoms,
                              const int *excl_off, const int *excl, const double4 *pos4,
                              const double *tq, Box box, double alpha, int apply_force,
                              long long *frc, long long *acc) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    double en = 0;
    if (m < nmol) {
        const int s = mol_off[m], e = mol_off[m + 1];
        const double a2 = alpha * alpha, a2pi = 2.0 * alpha / 1.7724538509055160273;
        for (int p = s; p < e; p++) {
            const int i = mol_atoms[p];
            const double4 pi = pos4[i];
            const double qi = tq[(int)pi.w];
            for (int q = p + 1; q < e; q++) {
                const int j = mol_atoms[q];
                bool ex = false;
                for (int k = excl_off[i]; k < excl_off[i + 1]; k++)
                    if (excl[k] == j) { ex = true; break; }
                if (!ex) continue;
                const double4 pj = pos4[j];
                double dx = pj.x - pi.x, dy = pj.y - pi.y, dz = pj.z - pi.z;
                pbc3(dx, dy, dz, box);
                const double r2 = dx * dx + dy * dy + dz * dz, r = sqrt(r2);
                const double qij = qi * tq[(int)pj.w];
                const double ee = erf(alpha * r) / r;
                en += qij * ee;
                if (apply_force) {
                    const double dudr = ee - a2pi * exp(-a2 * r2);
                    const double fs = qij * dudr / r2;
                    frc[i] += to_fix(fs * dx, FRC_SCALE);
                    frc[n + i] += to_fix(fs * dy, FRC_SCALE);
                    frc[2 * n + i] += to_fix(fs * dz, FRC_SCALE);
                    frc[j] -= to_fix(fs * dx, FRC_SCALE);
                    frc[n + j] -= to_fix(fs * dy, FRC_SCALE);
                    frc[2 * n + j] -= to_fix(fs * dz, FRC_SCALE);
                }
            }
        }
    }
    __shared__ double s_r[8];
    double t = warp_sum(en);
    if ((threadIdx.x & 31) == 0) s_r[threadIdx.x >> 5] = t;
    __syncthreads();
    if (threadIdx.x == 0) {
        double v = 0;
        for (int q = 0; q < (int)(blockDim.x >> 5); q++) v += s_r[q];
        if (v != 0.0) atomicAdd((unsigned long long *)&acc[ACC_E_INTRA], (unsigned long long)to_fix(-v, ACC_SCALE));
    }
}

void launch_intra(Ctx &c) {
    if (!c.ewald_on || !c.has_multisite) return;
    k_intra_ewald<<<(c.nmol + 127) / 128, 128, 0, c.stream>>>(
        c.nmol, c.n, c.mol_off, c.mol_atoms, c.excl_off, c.excl, c.pos4, c.type_q, c.box, c.ew_alpha,
        c.clen2 ? 0 : 1, c.frc, c.acc);  // constraints on: energy only
}

}  // namespace smd
