// Host-side context of one simulated system and the launchers of its kernels.
// The C-ABI in include/swinmd_b200.h hands callers an opaque pointer to this.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <string>
#include <type_traits>
#include <vector>
#include "smd_common.cuh"
#include "../../include/swinmd_b200.h"

namespace smd {

enum VdwKind { VDW_NONE = 0, VDW_LJ = 1, VDW_MIE = 2, VDW_BMH = 3, VDW_BUFF = 4, VDW_SAAP = 5 };

// surface-correction reduction: blocks of partial sums and sums per block
constexpr int CG_SCAL = 8;     // iterations, final RMS change, ...
constexpr int CG_TRACE = 64;   // RMS change of each iteration of the last solve
constexpr int SURF_BLOCKS = 64, SURF_SUMS = 11;

// Per type pair parameters of the short-range pair term (ntypes^2 rows of 8).
//   LJ : p0 sigma^2, p1 4 eps, p2 energy at the cutoff (shift), p3 unused
//   MIE: p0 sigma, p1 Cn*eps, p2 n, p3 m
//   BMH: p0 A, p1 1/rho, p2 C, p3 D
struct CellGrid {
    int use_cells;
    int n[3];
    int ncell;
    double len[3], rlen[3], origin[3];
    double L0[3];       // the box the grid was laid out for (the barostat scales it)
};

constexpr int LIST_GROUP = 8;   // sites per block of the list build

struct PairList {
    int max_nbr = 0;
    int *nbr = nullptr;      // [max_nbr][N]; bit 31 set = same molecule
    int *nnbr = nullptr;     // [N]
    int *cell_of = nullptr, *cell_count = nullptr, *cell_start = nullptr;
    unsigned *cell_slot = nullptr, *cell_fill = nullptr;
    int4 *cell_q = nullptr;  // the sites in cell order: box fractions, index
    int2 *group = nullptr;   // groups of up to LIST_GROUP sites of one cell: (cell, first slot)
    int *ngroup = nullptr;
    int cell_cap = 0;
    double rl2 = 0;          // (cutoff + cutBuff)^2
    double drmax = 0;        // cutBuff^2 / 4
};

constexpr int MP_SK_CHUNKS = 16;   // site chunks of the multipole structure factors at most
constexpr int MP_SK_BLOCK = 32;    // k per block of their reduction

struct Recip {               // Ewald reciprocal space (k half-space, k^2 < kcut^2)
    int nk = 0;
    int *kn = nullptr;       // [3][nk] integer lattice indices
    double *kcoef = nullptr; // [nk] 4 pi/V * exp(-k^2/4a^2)/k^2
    long long *sk = nullptr; // multipole passes: partial structure factors [MP_SK_CHUNKS][6][nk], totals
                             // [6][nk], block energies and virial [][8] (doubles)
    double *kvec = nullptr;  // [3][nk] k in 1/nm
    int nmax = 0;            // largest |n| of any component
    // sheared cell (SLLOD, point charges): the k list depends on the
    // Lees-Edwards offset, so it is (and its columns) are rebuilt on the device before every
    // evaluation; nk is then the candidate capacity and nk_dev the count
    int le = 0;
    int le_nx = 0, le_ny = 0, le_nz = 0;   // candidates nx 0..le_nx, ny - round(nx t) and nz within +-le_ny, +-le_nz
    int *nk_dev = nullptr;
    // point charges: the k set by columns (smd_recip.cu)
    int ew_cap = 0, ew_nx = 0, ew_ny = 0, ew_nzt = 8, ew_nch = 0, ew_chunks = 0;
    int4 *ew_col = nullptr;      // columns (nx, ny, largest nz, 0)
    int *ew_ncol = nullptr;      // live columns
    double *ew_part = nullptr;   // partial sums [chunks][nz][4][ew_cap]
    double4 *ew_coef = nullptr;  // force coefficients [ew_cap][nz]
    // FP32 passes of the polarisable model (built once per k set; the k list
    // is ordered column by column, nz ascending by one within a column)
    int nseg = 0, ncol = 0, row = 0, tab_n = 0;
    int4 *kseg = nullptr;    // runs of <= 4 k of one column (first k, count, nx | ny << 16, first nz)
    int4 *mcol = nullptr;    // columns (nx, ny, largest nz, 0)
    // column products, FP32 [0] and FP64 [1]: column groups, sites per chunk,
    // rows of blocks, the groups (first, count) and their (column, nz range) items
    int mblk[2] = {0, 0}, mchunk[2] = {0, 0}, mrows[2] = {0, 0};
    int2 *mgrp[2] = {nullptr, nullptr}, *mitem[2] = {nullptr, nullptr};
    void *mpart = nullptr;   // block totals [blocks][8], partial sums [rows][nz][8][items]
    void *mcoef[2] = {nullptr, nullptr};   // force coefficients [ncol][nz] of 4, FP32 and FP64
    float2 *stab = nullptr;  // per site phase tables [n][row]: e^{2 pi i m f / 2^32}, m < nmax + 1, per axis
    // the FP64 column passes: phase tables e^{2 pi i m f / 2^64} and FP64 site
    // records [n][4]
    double2 *stab_d = nullptr;
    double4 *srec_d = nullptr;
};

struct Ctx {
    int device = 0, sms = 1;   // and its multiprocessors
    cudaStream_t stream = nullptr;
    std::string err;
    // sizes
    int n = 0, nmol = 0, ntypes = 0;
    // host topology
    std::vector<int> h_type, h_mol, h_mol_off, h_mol_atoms, h_excl_off, h_excl;
    std::vector<double> h_mass, h_charge;
    std::vector<double> h_type_charge;
    double total_mass = 0;
    // device topology
    int *type = nullptr, *mol = nullptr, *mol_off = nullptr, *mol_atoms = nullptr;
    int *excl_off = nullptr, *excl = nullptr;
    double *mass = nullptr;
    double *pair_par = nullptr;    // [ntypes*ntypes*4]
    float *pair_par_f = nullptr;
    double *type_q = nullptr;      // scaled charge per type
    // state
    double4 *pos4 = nullptr, *vel4 = nullptr, *vtm4 = nullptr, *disp4 = nullptr;
    int4 *fixq = nullptr;
    long long *frc = nullptr;      // [3][N]
    long long *acc = nullptr;      // [ACC_COUNT]
    double *scal = nullptr;        // integrator scalars (see smd_integrate.cu)
    double *partials = nullptr;    // per-block reduction partials
    unsigned int *ticket = nullptr;
    unsigned int *status = nullptr;
    int *flags = nullptr;          // [0] rebuild list, [1] list builds so far, [2] stored dipole steps,
                                   // [3] their push's ticket, [4] the list build's ticket, [5] a site
                                   // is far outside the box
    smd_observables *obs = nullptr;  // observables of the last step, on device
    double *series = nullptr;      // recorded per-step samples
    int series_cap = 0;
    // configuration
    Box box{};
    CellGrid grid{};
    PairList pl;
    Recip rc;
    int precision = SMD_PREC_FP64;
    int reference_forms = 0;        // FP64 path: pow() buffered 14-7 and one sine/cosine per (site, k) reciprocal sums
    int want_cells = 1;
    // polarisable multipole model (Multipole / Induction / BuffvdWForce)
    int mp_on = 0, ind_on = 0;
    double mp_rc2 = 0;              // real-space cutoff^2 (cutoffEw)
    double ind_cut2 = 0;            // cutoffInd^2
    double thole_a = 0.39;
    int ind_amoeba = 0;              // induced real space: 0 Thole-damped B_n, 1 Tinker's AMOEBA form
    double *type_mp = nullptr;      // [ntypes][9] local dipole (3) + quadrupole (6)
    double *type_polar = nullptr;   // [ntypes] polarisabilities (nm^3)
    std::vector<double> h_type_polar;
    double *mu = nullptr;           // [3][N] lab-frame dipoles (e nm)
    double *qd = nullptr;           // [6][N] lab-frame quadrupoles (already /3)
    long long *trq = nullptr;       // [3][N] torques, fixed point
    double *e0 = nullptr;           // [3][N] permanent field at the sites
    double *pind = nullptr;         // [3][N] induced dipoles
    float4 *srec = nullptr;         // [N][4] mixed path, FP32: (q, mu), (Qxx, Qxy, Qxz, Qyy), (Qyz, Qzz, px, py), (pz, 0, 0, 0)
    double *cgw = nullptr;          // CG work: r, w, p [3][N] each, alpha [N], two gather copies [N][4], s, u [3][N]
    double *cgs = nullptr;          // CG scalars [CG_SCAL], trace [CG_TRACE], partials [4][blocks][4]
    int cg_max_iter = 500;
    double cg_tol = 2.0819e-8;      // RMS dipole change tolerance (e nm); 1e-6 D
    int cg_guess = 0;               // SMD_GUESS_*: 0 block solution of E0, 1 previous step, 2 learned, 3 first order
    int cg_blocks = 0;
    int pp_blocks = 0;              // grid of the pipelined solve (0: the layout does not allow it)
    size_t ps_smem = 0;             // the pipelined solve with the vector in shared memory: what a block may take
    int cg_pipelined = 1;           // pipelined solve (molecule blocks): 0 never, 1 mixed path, 2 both precisions
    int cg_precond = SMD_PRECOND_MOLECULE;  // dipole-solve preconditioner
    double *cg_blk = nullptr;       // [nmol][81] inverse molecule blocks of A
    unsigned int *cg_bar = nullptr; // grid barrier: [0] counter, [1] abort word of the launch
    unsigned long long wait_ns = 1000000000ull;  // limit of one device-side barrier wait (1 s)
    int test_skip_block = -1;       // failure-path test: solve block that never arrives
    int *ind_rj = nullptr;          // damped-tensor rows of the solve: partners [N][cap]
    void *ind_rc = nullptr;         // coefficients [N][cap] (float4 or double4)
    int *ind_cnt = nullptr;         // row lengths [N]
    int ind_cap = 0;
    double *phist = nullptr;        // last 4 steps' converged dipoles and fields [4][6][N] (ring, count in flags[2])
    int in_step = 0;                // enqueueing the step graph: the solve stores its dipoles
    double *frame = nullptr;        // [9][N] site axes u, v, w (lab frame)
    // per-site network giving the initial induced dipoles (smd_mlp.cu)
    int mlp_ready = 0;
    int mlp_base = 2;                // order of the extrapolated guess the network corrects
    int mlp_tc = 1;                  // inference and evaluation: 1 tcgen05 tiles of 128 rows, 0 warp-level mma.sync
    float *mlp_w = nullptr;         // parameters, MLP_NPARAM floats
    float *mlp_m = nullptr, *mlp_v = nullptr;  // Adam moments
    float *mlp_part = nullptr;      // per-block gradient partials
    float *mlp_norm = nullptr;      // feature mean [F] and 1/std [F]
    float *mlp_x = nullptr;         // [N][F] raw features of the current configuration
    float *mlp_data = nullptr;      // training rows [cap][F + 3]
    long long mlp_rows = 0, mlp_cap = 0;
    int mlp_t = 0;                  // Adam step count
    // buffered 14-7 with virtual H sites
    int buff_on = 0;
    double buff_n = 14, buff_m = 7, buff_delta = 0.07, buff_gamma = 0.12, buff_h = 0.91;
    double buff_c[6] = {0, 0, 0, 0, 0, 0};
    double buff_sw = 0;             // taper start (nm)
    double4 *vpos4 = nullptr;       // virtual site positions
    int4 *vfixq = nullptr;          // their 32-bit box fractions
    long long *fv = nullptr;        // [3][N] forces on the virtual sites
    int has_multisite = 0;          // some molecule has more than one site
    int mol_sites = 0;              // sites per molecule when molecule m's are mol_sites m .. mol_sites m + mol_sites - 1 for every m, else 0
    // bonded terms of flexible molecules (smd_bonded.cu)
    int nbond = 0, nangle = 0, bond_form = 1, ub_on = 0;
    double ub_k = 0, ub_l0 = 0;
    int4 *bonds = nullptr;          // (atom1, atom2, type, 0)
    int4 *angles = nullptr;         // (atom1, atom2, atom3, type)
    double2 *bond_par = nullptr;    // per type (r0, k)
    double2 *angle_par = nullptr;   // per type (theta0, k)
    // radial distribution function (smd_rdf.cu)
    int rdf_nbins = 0;
    long long rdf_samples = 0;
    double rdf_maxr = 0;
    unsigned long long *rdf_hist = nullptr;  // [ntypes][ntypes][nbins]
    int excl_intermol = 0;          // some exclusion joins two molecules
    // Atom::realPos bookkeeping: box shifts per molecule since the last
    // position upload, and the uploaded offsets realPos - position
    double *wrap = nullptr;         // [3][nmol]
    std::vector<double> h_real_off; // [3N] (empty: realPos = position at upload)
    // running averages of the step observables (smd_integrate.cu)
    double *avg = nullptr;          // [AVG_COUNT] sums, updated by every step
    // surface-dipole corrections (smd_surface.cu)
    int surface_on = 0;
    double *surf_part = nullptr;    // per-block partial sums
    double *surf_tot = nullptr;     // the sums
    double *clen2 = nullptr;        // [nmol][3] squared SHAKE distances
    int fixq_from_integrate = 0;    // step graph: integrate writes fixq
    int vdw = VDW_NONE;
    double cutoff = 1.0, cut_buffer = 0.1;
    double vdw_rc2 = 1.0, sw_rs2 = 0.0, sw_c1 = 0, sw_c2 = 0, sw_c3 = 0;
    int switch_on = 0;
    double e_lrc = 0, v_lrc = 0;
    double *saap = nullptr;         // SAAP pair parameters a0..a5 per type pair
    // Wolf summation of the charges (WolfForce)
    int wolf_on = 0;
    double wolf_alpha = 0, wolf_rc = 0, wolf_d = 0;
    int wolf_msites = 0;            // some charge sits on a displaced site
    int *wolf_msite = nullptr;      // per site: 1 if its charge is displaced
    double4 *wpos4 = nullptr;       // charge-site positions
    // isotropic barostat of the chain integrator (NHIntegrator's NpT run)
    int npt = 0;
    double npt_press = 0;           // target pressure, kJ/mol/nm^3
    double npt_tau = 0;             // BarosConst (ps)
    double npt_lrc_k = 0;           // tail-correction energy x volume
    double npt_smin = 0;            // smallest box scale the cell grid covers
    Box *dbox = nullptr;            // the box on the device while the barostat runs
    int ewald_on = 0;
    double ew_alpha = 0, ew_kcut = 0, ew_rc2 = 0, e_self = 0;
    int long_steps = 1;
    smd_integrator_params ip{};
    int integrator_ready = 0;
    int tpp = 0;                    // threads per site in the pair kernel (0: lanes_per_site)
    int nb_blocks = 0;              // blocks of the integrate kernel
    long long steps_done = 0;
    int list_valid = 0;
    int list_built = 0;      // a pair list exists for the current set-up (its sites may have moved within the skin)
    double *stage = nullptr;     // [3][n][3] staging of uploaded and downloaded positions, velocities and v-
    double *fout = nullptr;      // [3N] device force output of smd_compute_forces, allocated once
    // configuration version: bumped by every call that moves the sites or
    // changes the model or the solver; smd_compute_forces solves the induced
    // dipoles only when they were not solved for the current version
    long long cfg_version = 1;
    long long dip_version = 0;
    // scratch of the on-demand volume derivatives (smd_lustig.cu)
    double4 *lus_com = nullptr;     // [nmol] molecular centres of mass
    double *lus_buf = nullptr;      // per-block / per-k partial sums
    size_t lus_cap = 0;
    // CUDA graph of one step
    cudaGraphExec_t step_graph = nullptr;
    int graph_dirty = 1;
};

// e^{x^2} erfc(x), x >= 0: (x + 2) erfcx(x) as a polynomial in u = (x - 2)/(x +
// 2) (the variable of M. M. Shepherd and J. G. Laframboise, Math. Comp. 36 (1981)
// 249), interpolated at the Chebyshev nodes of 0 <= x <= 12 in 50 digits to
// 3e-17; in FP64 1.3e-16 rms, at most 4e-16.  Past 12 it multiplies an
// exponential below 1e-62.  Even and odd powers run as two chains.  With
// gauss_of the real-space terms share one exponential where they took erfc and
// exp, and carry the exponent's rounding, which those amplify by 2 x^2: force
// factor against 30 digits 1.2e-16 to 1.6e-16 rms for a = 2.8 to 9 and r up to
// 1.2 (2.5e-16 to 2.3e-15 with erfc and exp).  FP64 LJ + Ewald 30.4 -> 25.4 us
// at 2331 sites, multipoles 115 -> 106 and induced 134 -> 124 at 3993.
__device__ __forceinline__ double erfcx_pos(double x) {
    constexpr double c[23] = {1.021582705242023, -0.6871606844138112, 0.27947209255606176, -0.0364422315068082,
        -0.0215106618899279, 0.006479185065065647, 0.0030906120698213097, -0.0008372960141435824,
        -0.0006630736335767911, 3.43709343512164e-05, 0.0001444716182169992, 3.415216055606241e-05,
        -2.1699632130063324e-05, -1.6134777250867785e-05, -1.1184215188592036e-06, 3.682673067728124e-06,
        1.9981025544757337e-06, -6.902304551418623e-08, -5.882578109581312e-07, -2.4385788675464163e-07,
        3.9988998520065743e-08, 6.063779704411114e-08, 1.413518017460013e-08};
    const double v = 1.0 / (x + 2.0), u = fma(-4.0, v, 1.0), u2 = u * u;
    double e = c[22], o = c[21];
#pragma unroll
    for (int q = 20; q >= 0; q -= 2) {
        e = fma(e, u2, c[q]);
        if (q > 0) o = fma(o, u2, c[q - 1]);
    }
    return fma(o, u, e) * v;
}
// e^{-a^2 r^2} with the exponent's rounding carried
__device__ __forceinline__ double gauss_of(double a, double r2) {
    const double a2 = a * a, z = a2 * r2;
    const double ex = exp(-z);
    return fma(ex, -(fma(a2, r2, -z) + fma(a, a, -a2) * r2), ex);
}

// Lanes that share one site's list row in the pair-type kernels.  A row is
// walked serially by its lanes, so few sites want many lanes (the chip is
// empty and the walk is the time), while short rows of many sites want few
// (the lanes' reduction and idle last pass cost more than the walk).  B200,
// us for 4 / 8 / 16 / 32 lanes: FP64 LJ (78 entries a row) 2048 sites 12.9 /
// 8.2 / 5.9 / 6.2, 16384 15.4 / 18.5 / 20.7 / 29.4, 62500 42.8 / 46.0 / 57 /
// 91; FP64 LJ + Ewald (560 entries) 2331 sites 163 / 84 / 45 / 30, 6480 156 /
// 102 / 88 / 82, 12000 197 / 169 / 150 / 148; mixed LJ + Ewald 2331 sites 64 /
// 34 / 20 / 14, 6480 63 / 42 / 32 / 33; mixed fused polarisable pass (300
// entries, 8 / 16 / 32 lanes) 1029 sites 65 / 37 / 26, 3993 85 / 87 / 83,
// 12288 210 / 203 / 211.
inline int lanes_per_site(const Ctx &c) {
    const double rl = c.cutoff + c.cut_buffer, vol = c.box.L[0] * c.box.L[1] * c.box.L[2];
    const double entries = vol > 0 ? 4.18879 * rl * rl * rl * c.n / vol : 0.0;
    if (c.n <= 2600) return 32;
    if (entries >= 128) return 16;
    return c.n <= 8000 ? 16 : (c.n <= 12000 ? 8 : 4);
}

// the same for the kernels built for 8, 16 and 32 lanes, and a call of f with
// that count as a compile-time constant
inline int wide_lanes(const Ctx &c) {
    const int l = lanes_per_site(c);
    return l < 8 ? 8 : l;
}
template <class F>
inline void with_lanes(int tpp, F f) {
    if (tpp >= 32) f(std::integral_constant<int, 32>());
    else if (tpp >= 16) f(std::integral_constant<int, 16>());
    else f(std::integral_constant<int, 8>());
}

// launchers (each enqueues on ctx.stream)
void launch_fixq(Ctx &c);
void launch_put_positions(Ctx &c, bool keep_list);
void launch_put_velocities(Ctx &c, bool own_vtm);
void launch_get_state(Ctx &c, bool pos, bool vel, bool vtm);
void launch_nlist(Ctx &c, bool force_rebuild);
void launch_pair(Ctx &c);
void launch_recip(Ctx &c);
void launch_integrate(Ctx &c);
void launch_start_velocities(Ctx &c);
void launch_nhc_first(Ctx &c);
void launch_nhc_second(Ctx &c);
void launch_nhc_start(Ctx &c);
void launch_finalize_forces(Ctx &c, double *f_out_dev);
void launch_intra(Ctx &c);
// polarisable model: term groups (each maps its own torques to forces)
void launch_mp_short(Ctx &c);
void launch_mp_long(Ctx &c);
void launch_ind_solve(Ctx &c);
void launch_ind_field(Ctx &c);
void launch_ind_cg(Ctx &c);
void launch_ind_short(Ctx &c);
void launch_mp_mol(Ctx &c);
bool polar_short_fused(const Ctx &c);
void launch_polar_short(Ctx &c);
inline void touch(Ctx &c) { c.cfg_version++; }
void launch_ind_long(Ctx &c);
void launch_polar_long(Ctx &c);
void launch_torques_end(Ctx &c);
void launch_frames(Ctx &c);
void launch_bonded(Ctx &c, bool bond, bool angle, bool ub);
void launch_intra_flex(Ctx &c, bool mp, bool ind);
int rdf_sample(Ctx &c);
void launch_surface(Ctx &c, bool ewald, bool mp, bool ind);
inline bool has_bonded(const Ctx &c) { return c.nbond > 0 || c.nangle > 0 || c.ub_on; }

// Running sums of the step observables (the energy and stress averages of
// Ensemble::accumulate, src/Ensemble.cpp:814-894), added by the last block
// of every step, in the layout of smd_averages after its sample count:
// [0] samples, [1..11] energies, [12..21] atomic and molecular stress,
// [22..39] atomic and molecular pressure tensors.  One thread per sum takes
// its term of the finished observables: one thread adding all 40 waits 40
// dependent round trips to L2 (10 us of a step).
constexpr int AVG_COUNT = 40;
__device__ __forceinline__ double average_term(int q, const smd_observables &o) {
    const double et = o.e_potential + o.ke_atom;
    if (q >= 22) return q < 31 ? o.atom_pressure[q - 22] : o.mol_pressure[q - 31];
    if (q >= 12) {
        const double *p = q < 17 ? o.atom_pressure : o.mol_pressure;
        switch (q < 17 ? q - 12 : q - 17) {
            case 0: return (p[0] + p[4] + p[8]) / 3.0;
            case 1: return (p[1] + p[3]) * 0.5;   // shear stress (XY + YX) / 2
            case 2: return (p[3] - p[1]) * 0.5;   // antisymmetric part (YX - XY) / 2
            case 3: return p[0] - p[4];           // first normal stress difference
            default: return p[4] - p[8];          // second normal stress difference
        }
    }
    switch (q) {
        case 0: return 1.0;
        case 1: return o.e_potential;
        case 2: return o.e_potential * o.e_potential;
        case 3: return et;
        case 4: return et * et;
        case 5: return o.ke_atom;
        case 6: return o.ke_atom * o.ke_atom;
        case 7: return o.ke_mol;
        case 8: return o.ke_mol * o.ke_mol;
        case 9: return o.ke_mol != 0.0 ? 1.0 / o.ke_mol : 0.0;
        case 10: return o.volume;
        default: return o.volume * o.volume;
    }
}

// What the last block of a step reads besides the partial sums and hands out
// again, through shared memory: loaded by many threads at once before the
// totals, written by many threads after them.
struct StepTail {
    long long acc[ACC_COUNT];
    smd_observables o;
    long long step;          // steps before this one
    int list_updates;
    unsigned int status;
    double scal[SC_NSCAL];
};
static_assert(sizeof(smd_observables) % 8 == 0, "copied in 8-byte words");

// the averages' old value of thread t (t < AVG_COUNT), and the rest of
// the tail's inputs into s
__device__ __forceinline__ double tail_load(StepTail &s, int t, int nt, const long long *acc, const double *avg,
                                            const double *scal, const smd_observables *obs, const int *flags,
                                            const unsigned int *status) {
    for (int q = t; q < ACC_COUNT; q += nt) s.acc[q] = __ldcg(&acc[q]);
    for (int q = t; q < SC_NSCAL; q += nt) s.scal[q] = __ldcg(&scal[q]);
    if (t == nt - 1) s.step = __ldcg((const long long *)&obs->step);
    if (t == nt - 2) s.list_updates = __ldcg(&flags[1]);
    if (t == nt - 3) s.status = __ldcg(status);
    return avg && t < AVG_COUNT ? __ldcg(&avg[t]) : 0.0;
}

// the finished observables, averages (old: tail_load's value), the step's
// sample of the series, and cleared accumulators and ticket
__device__ __forceinline__ void tail_store(const StepTail &s, int t, int nt, double old, long long *acc, double *avg,
                                           smd_observables *obs, double *series, int series_cap, double sample4,
                                           unsigned int *ticket) {
    const long long *src = (const long long *)&s.o;
    for (int q = t; q < (int)(sizeof(smd_observables) / 8); q += nt) ((long long *)obs)[q] = src[q];
    if (avg && t < AVG_COUNT) avg[t] = old + average_term(t, s.o);
    if (series_cap > 0 && t == nt - 1) {
        double *r = series + (s.o.step - 1) % series_cap * 5;
        r[0] = s.o.e_potential; r[1] = s.o.ke_atom; r[2] = s.o.t_atom; r[3] = s.o.zeta; r[4] = sample4;
    }
    for (int q = t; q < ACC_COUNT; q += nt) acc[q] = 0;
    if (t == nt - 2) *ticket = 0;
}

// Sums of NP values per lane over the warp, value q left in dst[q]: the
// first 32 by a transposed butterfly (each step exchanges half of what is
// left, 31 exchanges in place of 32 x 5), the rest by plain ones.  Fixed
// order, so the result is the same on every run.
template <int NP>
__device__ __forceinline__ void warp_sum_many(const double (&part)[NP], double *dst) {
    const int lane = threadIdx.x & 31;
    double v[32];
#pragma unroll
    for (int q = 0; q < 32; q++) v[q] = q < NP ? part[q < NP ? q : 0] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int q = 0; q < o; q++) {
            if (q >= NP) continue;
            const double send = up ? v[q] : v[q + o], keep = up ? v[q + o] : v[q];
            v[q] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    if (lane < NP) dst[lane] = v[0];
#pragma unroll
    for (int q = 32; q < NP; q++) {
        const double x = warp_sum(part[q < NP ? q : 0]);
        if (lane == 0) dst[q] = x;
    }
}

// the energy components of the accumulator slots (energy[SMD_E_COUNT]);
// e_lrc and e_self are the constant tail and self energies added to the
// vdW and self slots
__host__ __device__ inline void acc_energies(const long long *acc, double e_lrc, double e_self, double *en) {
    for (int q = 0; q < SMD_E_COUNT; q++) en[q] = 0.0;
    en[SMD_E_VDW] = (double)acc[ACC_E_VDW] * ACC_INV + e_lrc;
    en[SMD_E_REAL] = (double)acc[ACC_E_REAL] * ACC_INV;
    en[SMD_E_LONG] = (double)acc[ACC_E_LONG] * ACC_INV;
    en[SMD_E_CORRECT] = e_self + (double)acc[ACC_E_SELF] * ACC_INV;
    en[SMD_E_MOLCORRECT] = (double)acc[ACC_E_INTRA] * ACC_INV;
    en[SMD_E_SURF] = (double)acc[ACC_E_SURF] * ACC_INV;
    en[SMD_E_POL_REAL] = (double)acc[ACC_E_POL_REAL] * ACC_INV;
    en[SMD_E_POL_LONG] = (double)acc[ACC_E_POL_LONG] * ACC_INV;
    en[SMD_E_POL_SELF] = (double)acc[ACC_E_POL_SELF] * ACC_INV;
    en[SMD_E_POL_INTRA] = (double)acc[ACC_E_POL_INTRA] * ACC_INV;
    en[SMD_E_POL_SURF] = (double)acc[ACC_E_POL_SURF] * ACC_INV;
    en[SMD_E_BOND] = (double)acc[ACC_E_BOND] * ACC_INV;
    en[SMD_E_ANGLE] = (double)acc[ACC_E_ANGLE] * ACC_INV;
    en[SMD_E_UB] = (double)acc[ACC_E_UB] * ACC_INV;
}
void launch_buff(Ctx &c);
int setup_cg(Ctx &c);
int solve_grid(const Ctx &c);   // blocks of the dipole solve that the present settings choose
void solve_layout(const Ctx &c, int32_t *layout);   // its form, blocks and held slots (smd_solver_layout)
int recip_nk(Ctx &c, int *nk);
int ensure_ind_rows(Ctx &c);
// dipole-guess network (smd_mlp.cu)
int mlp_alloc(Ctx &c, long long cap_rows, unsigned int seed);
void launch_mlp_guess(Ctx &c);
void launch_first_order_guess(Ctx &c);
void launch_blk_response(Ctx &c, double *out, int order, double *out_prev);
int lustig_lj(Ctx &c, double *out);
int lustig_all(Ctx &c, double *out);
void launch_wolf_sites(Ctx &c);
void launch_mp_real_only(Ctx &c);
void launch_ind_real_only(Ctx &c);
void launch_ind_self_only(Ctx &c);
void launch_intra_flex_lus(Ctx &c, bool mp, bool ind, double *fr_mol);
// order of the extrapolated guess of the solver's guess mode (0: none)
inline int guess_order(const Ctx &c) {
    return c.cg_guess == SMD_GUESS_FIRST_ORDER ? 1
           : c.cg_guess == SMD_GUESS_EXTRAP2   ? 2
           : c.cg_guess == SMD_GUESS_EXTRAP3   ? 3
                                               : 0;
}
// first-order part of the learned guess: the solver's s slot of its work
// area, which the solve writes before it first reads it
inline double *guess_response(Ctx &c) { return c.cgw + 20 * (size_t)c.n; }
// M^-1 (E0(t-1) - E0(t-2)), the network's input (the solve's residual
// buffer, free until the solve starts)
inline double *guess_response_prev(Ctx &c) { return c.cgw; }
int mlp_batch_loss(Ctx &c, const unsigned int *perm, int batch, double *loss);
void launch_mlp_features(Ctx &c);
void launch_mlp_collect(Ctx &c);
void launch_mlp_norm(Ctx &c);
void launch_mlp_step(Ctx &c, const unsigned int *perm, long long r0, int batch, float lr, float *grad_out);
void launch_mlp_eval(Ctx &c, int rows, const float *x, float *y);
int mlp_nparam();
int mlp_nfeat();
int mlp_max_batch();
int setup_recip(Ctx &c);
int mp_recip_prepare(Ctx &c);

}  // namespace smd
