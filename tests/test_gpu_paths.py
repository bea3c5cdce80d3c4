"""Kernels whose shape follows the system's size: the point-charge reciprocal
columns, the list build, the lanes per site and the dipole solve, at the
edges of their ranges, against plain FP64 sums or the form next to them."""
import numpy as np
import pytest

from conftest import rms_rel
from swinmd_b200 import engine, systems
from swinmd_b200 import _lib as L

pytestmark = pytest.mark.gpu


def _ewald_direct(s, box, alpha, kcut):
    m = int(kcut * box / (2 * np.pi))
    g = np.arange(-m, m + 1)
    n = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    half = (n[:, 0] > 0) | ((n[:, 0] == 0) & ((n[:, 1] > 0) | ((n[:, 1] == 0) & (n[:, 2] > 0))))
    k = n[half] * (2 * np.pi / box)
    k2 = (k * k).sum(1)
    k, k2 = k[k2 < kcut ** 2], k2[k2 < kcut ** 2]
    c = 4 * np.pi / box ** 3 * np.exp(-k2 / (4 * alpha ** 2)) / k2
    q, ph = s.scaled_charges(), s.pos @ k.T
    sn, cs = np.sin(ph), np.cos(ph)
    C, S = q @ cs, q @ sn
    return q[:, None] * ((2 * c * (sn * C - cs * S)) @ k), float((c * (C * C + S * S)).sum()), len(k)


# columns of 3 .. 17 nz: each item length (5 to 8) with one to three items
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("kmax", [3, 5, 6, 7, 8, 9, 10, 13, 17])
def test_ewald_columns(kmax, precision):
    s = systems.nacl_melt(ncell=8, kmax=kmax, seed=2)
    ens = engine.GpuEnsemble(s, precision=precision)
    f, e, _ = ens.compute_forces(L.TERM_EWALD_LONG)
    fr, er, nk = _ewald_direct(s, ens.box, s.config.alpha, s.config.k_cutoff)
    assert ens.ewald_nk() == nk
    # forces of 1e2 kJ/mol/nm in units of 2^-32, FP64 throughout
    assert rms_rel(f, fr) < 1e-11
    assert abs(e[L.E_LONG] - er) < 1e-10 * abs(er)
    ens.close()


# sites uploaded outside the box keep the reference's cell rule: the nearest
# cell, and no minimum image inside a cell
@pytest.mark.parametrize("share,boxes", [(0.0, 0), (0.05, 1), (0.3, 2)])
@pytest.mark.parametrize("ncell", [5, 8, 9])
def test_pair_list_of_unwrapped_positions(ncell, share, boxes):
    s = systems.lj_fluid(ncell=ncell, seed=4, jitter_star=0.1)
    rng = np.random.default_rng(ncell)
    ens = engine.GpuEnsemble(s)
    box, rl = ens.box, s.config.cutoff + s.config.cut_buffer
    pos = s.pos + box * np.where(rng.random(s.pos.shape) < share, rng.integers(-boxes, boxes + 1, s.pos.shape), 0)
    ens.upload_positions(pos)
    got = ens.pairs()
    nc = int(box / rl) if rl <= box / 3 else 0
    i, j = np.triu_indices(s.n_atoms, 1)
    d = pos[j] - pos[i]
    wrapped = d.copy()
    for _ in range(8):
        wrapped = np.where(wrapped >= box / 2, wrapped - box, wrapped)
    for _ in range(8):
        wrapped = np.where(wrapped < -box / 2, wrapped + box, wrapped)
    near = np.ones(len(i), bool)
    if nc:
        c = np.clip(((pos + box / 2) * (1.0 / (box / nc))).astype(int), 0, nc - 1)
        dc = (c[j] - c[i]) % nc
        near = ((dc <= 1) | (dc == nc - 1)).all(1)
        wrapped = np.where((c[i] == c[j]).all(1)[:, None], d, wrapped)
    take = near & ((wrapped ** 2).sum(1) < rl * rl)
    want = np.stack([i[take], j[take]], 1)
    got = got[np.lexsort((got[:, 1], got[:, 0]))]
    assert np.array_equal(got, want)
    ens.close()


# either side of the lane rule's lines (2600, 8000, 24000 sites)
@pytest.mark.parametrize("ncell", [8, 9, 12, 13, 18, 19])
def test_lanes_per_site(ncell):
    s = systems.lj_fluid(ncell=ncell, seed=6, jitter_star=0.08)
    f = []
    for tpp in (0, 8):
        ens = engine.GpuEnsemble(s, threads_per_site=tpp)
        f.append(ens.compute_forces()[0])
        ens.close()
    # sums of the same FP64 terms in another order, in units of 2^-32
    assert rms_rel(f[0], f[1]) < 1e-11


# 32, 16 and 8 lanes per site in the solve with the vector in shared memory,
# all or part of the rows held there, and the first size past it
@pytest.mark.parametrize("nmol", [343, 1184, 1185, 2368, 2369, 4500])
def test_dipole_solve_shapes(nmol):
    s = systems.polarizable_water(nmol=nmol, kmax=6, seed=5)
    ens = engine.GpuEnsemble(s, precision="mixed")
    p, it = [], []
    for mode in (0, 1):
        ens.set_solver_pipelined(mode)
        ens.compute_forces(L.TERM_IND_SHORT)
        p.append(ens.polarization()["p"])
        it.append(ens.solver_stats()[0])
    # both stop below an RMS change of 2.08e-8 e nm, and an iteration takes
    # the error down by 4.5, so each is within 0.3 of that of the solution
    assert np.sqrt(((p[0] - p[1]) ** 2).mean()) < 2.0819e-8
    assert abs(it[0] - it[1]) <= 1
    ens.close()


# column products of the multipole reciprocal sums: every width of the force
# pass's tables (8, 12, 16, 20, 32 nz) and the k sets past them
@pytest.mark.parametrize("kmax", [5, 8, 9, 12, 13, 16, 17, 20, 21, 32, 33])
def test_multipole_columns(kmax):
    s = systems.polarizable_water(nmol=216, cutoff=0.9, switch=0.8, kmax=kmax, seed=7)
    terms = L.TERM_MP_SHORT | L.TERM_MP_LONG | L.TERM_IND_SHORT | L.TERM_IND_LONG
    ens = engine.GpuEnsemble(s)
    ens.set_solver(tol=1e-13, max_iter=1000)
    ens.set_reference_forms(True)      # one FP64 sine and cosine per (site, k)
    ref = [ens.compute_forces(t) for t in (terms, L.TERM_MP_LONG)]
    for precision, tol in (("fp64", 1e-10), ("mixed", 1e-6)):
        ens.set_precision(precision)
        ens.set_reference_forms(False)
        for (f, e, w), t in zip(ref, (terms, L.TERM_MP_LONG)):
            fm, em, wm = ens.compute_forces(t)
            assert rms_rel(fm, f) < tol
            for q in (L.E_LONG, L.E_POL_LONG):
                assert abs(em[q] - e[q]) <= tol * abs(e[q])
            assert np.abs(wm - w).max() < tol * np.abs(w).max()
    ens.close()


# the FP32 Ewald pair term from x = alpha r < 1 to far past the polynomials'
# range.  Ten roundings of 2^-24 a pair, and a net force a third of its pairs'
@pytest.mark.parametrize("alpha", [0.5, 3.1, 9.0, 20.0, 150.0])
def test_ewald_pair_range(alpha):
    s = systems.spce_water(nmol=343, box=2.4, alpha=alpha, seed=5)
    ens = engine.GpuEnsemble(s)
    f = []
    for precision in ("fp64", "mixed"):
        ens.set_precision(precision)
        f.append(ens.compute_forces(L.TERM_EWALD_REAL)[0])
    assert np.isfinite(f[1]).all()
    rms = lambda x: np.sqrt((x ** 2).mean())   # noqa: E731
    assert rms(f[1] - f[0]) < 2e-6 * rms(f[0]) + 1e-8   # forces are held in 2^-32
    ens.close()


# k sets of a few columns, whose rows are shorter than one batch of the force
# pass's loads, after a kernel that leaves NaN in the multiprocessors' shared
# memory (a product of NaN matrices): what a load finds past the last column's
# row must not enter.  Bounds as in test_multipole_columns
@pytest.mark.parametrize("kmax", [2, 3])
def test_multipole_columns_few(kmax):
    import torch
    s = systems.polarizable_water(nmol=1331, cutoff=0.9, switch=0.8, kmax=kmax, seed=7)
    nan = torch.full((4096, 4096), float("nan"), dtype=torch.float64, device="cuda")
    ens = engine.GpuEnsemble(s)
    ens.set_reference_forms(True)
    fr, er, wr = ens.compute_forces(L.TERM_MP_LONG)
    for precision, tol in (("fp64", 1e-10), ("mixed", 1e-6)):
        ens.set_precision(precision)
        ens.set_reference_forms(False)
        nan @ nan
        torch.cuda.synchronize()
        f, e, w = ens.compute_forces(L.TERM_MP_LONG)
        assert np.isfinite(f).all()
        assert rms_rel(f, fr) < tol
        assert abs(e[L.E_LONG] - er[L.E_LONG]) <= tol * abs(er[L.E_LONG])
        assert np.abs(w - wr).max() < tol * np.abs(wr).max()
    ens.close()


# a box without cells and more sites than one stage of the build, one of the
# late ones uploaded 10 boxes away: the minimum image takes 8 steps at most
# (which leaves it 2 boxes from everything), in both rows of every pair
@pytest.mark.parametrize("site", [3, 1300])
def test_pair_list_without_cells_far_site(site):
    s = systems.lj_fluid(ncell=7, seed=4, jitter_star=0.1)
    s.config.use_cell_list = False
    ens = engine.GpuEnsemble(s, precision="mixed")
    pos = s.pos.copy()
    pos[site, 0] += 10 * ens.box
    ens.upload_positions(pos)
    p = ens.pairs()
    assert not (p == site).any()
    f, _, _ = ens.compute_forces()
    assert not f[site].any()
    # pair forces of 1e3 to 1e4 kJ/mol/nm, each side in FP32: 1e-7 of that a pair
    assert np.abs(f.sum(0)).max() < 1e-2
    ens.close()


# the column products' workspace: at most 512 MB of partial sums, the site
# tables (96 entries of 8 and of 16 bytes and a record of 128 bytes a site) and
# coefficients and items below 32 MB; the k set past the tables (kmax 33) takes
# none of it.  Past that size the sums go in several launches
def test_multipole_columns_workspace():
    import torch
    free = lambda: torch.cuda.mem_get_info()[0]   # noqa: E731
    s = systems.polarizable_water(nmol=20000, cutoff=0.9, switch=0.8, kmax=32, seed=7)
    n, k32 = s.n_atoms, s.config.k_cutoff
    torch.zeros(1, device="cuda")
    used = []
    for kcut in (k32 * np.sqrt((33 ** 2 - 0.5) / (32 ** 2 - 0.5)), k32):
        s.config.k_cutoff = kcut
        before = free()
        ens = engine.GpuEnsemble(s)
        used.append(before - free())
        if kcut > k32:
            ens.close()
    assert used[1] - used[0] < (512 << 20) + n * (96 * 24 + 128) + (32 << 20)
    ens.set_reference_forms(True)
    fr, er, _ = ens.compute_forces(L.TERM_MP_LONG)
    ens.set_reference_forms(False)
    for precision, tol in (("fp64", 1e-10), ("mixed", 1e-6)):
        ens.set_precision(precision)
        f, e, _ = ens.compute_forces(L.TERM_MP_LONG)
        assert rms_rel(f, fr) < tol
        assert abs(e[L.E_LONG] - er[L.E_LONG]) <= tol * abs(er[L.E_LONG])
    ens.close()


# the point-charge reciprocal energy is rounded to its 2^-28 kJ/mol once; a few
# FP64 roundings a term beside it
@pytest.mark.parametrize("kmax", [9, 13, 17])
def test_ewald_energy_rounding(kmax):
    s = systems.nacl_melt(ncell=8, kmax=kmax, seed=2)
    ens = engine.GpuEnsemble(s)
    _, e, _ = ens.compute_forces(L.TERM_EWALD_LONG)
    _, er, _ = _ewald_direct(s, ens.box, s.config.alpha, s.config.k_cutoff)
    assert abs(e[L.E_LONG] - er) < 2.0 ** -29 + 1e-13 * abs(er)
    ens.close()


# either side of the lane rule's lines as they are (2600, 8000 and 12 000 sites),
# against two lanes per site, which the rule never takes
@pytest.mark.parametrize("kind,size,precision", [("lj", 8, "fp64"), ("lj", 9, "fp64"), ("lj", 12, "fp64"),
                                                 ("lj", 13, "fp64"), ("lj", 14, "fp64"), ("lj", 15, "fp64"),
                                                 ("lj", 14, "mixed"), ("lj", 15, "mixed"), ("spce", 866, "fp64"),
                                                 ("spce", 867, "fp64"), ("spce", 866, "mixed"),
                                                 ("spce", 867, "mixed")])
def test_lanes_per_site_lines(kind, size, precision):
    s = (systems.lj_fluid(ncell=size, seed=6, jitter_star=0.08) if kind == "lj" else
         systems.spce_water(nmol=size, box=4.03 * (size / 2160) ** (1 / 3), seed=6, kmax=6))
    f = []
    for tpp in (0, 2):
        ens = engine.GpuEnsemble(s, precision=precision, threads_per_site=tpp)
        f.append(ens.compute_forces(L.TERM_VDW | L.TERM_EWALD_REAL)[0])
        ens.close()
    # sums of the same terms in another order, in units of 2^-32: FP64, and FP32
    # of up to 280 terms a lane
    assert rms_rel(f[0], f[1]) < (1e-11 if precision == "fp64" else 1e-6)


# the polarisable kernels with 32 and with 16 lanes a site: mixed against FP64
@pytest.mark.parametrize("nmol", [866, 867])
def test_lanes_per_site_polarisable(nmol):
    s = systems.polarizable_water(nmol=nmol, kmax=6, seed=5)
    ens = engine.GpuEnsemble(s)
    ens.set_solver(tol=1e-13, max_iter=1000)
    f = []
    for precision in ("fp64", "mixed"):
        ens.set_precision(precision)
        f.append([ens.compute_forces(t)[0] for t in (L.TERM_VDW, L.TERM_MP_SHORT, L.TERM_IND_SHORT, L.TERM_ALL)])
    for a, b in zip(*f):
        assert rms_rel(b, a) < 1e-6
    ens.close()
