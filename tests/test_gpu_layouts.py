"""Boxes with three different edges and sites in another order than molecule
by molecule: the list build, the reciprocal columns and the integrators, whose
kernels carry three edges and index molecules directly where they can."""
import numpy as np
import pytest

import oracle
from conftest import rms_rel
from swinmd_b200 import engine, systems
from swinmd_b200 import _lib as L

pytestmark = pytest.mark.gpu

EDGES = np.array([0.9, 1.0, 1.15])


def _three_edges(s, **kw):
    """An ensemble of s with the box edges and the molecules' centres scaled by
    EDGES (the molecules stay as they are)."""
    box = np.array(s.box) * EDGES
    first = np.unique(s.mol_id, return_index=True)[1][s.mol_id]
    near = s.pos - s.pos[first]
    near -= s.box[0] * np.round(near / s.box[0])
    pos = s.pos[first] * EDGES + near
    ens = engine.GpuEnsemble(s, **kw)
    ens._chk(ens.lib.smd_set_box(ens.ctx, *box))
    ens.upload_positions(pos)
    return ens, pos, box


# without cells, with cells (4, 4, 5), (6, 7, 8)
@pytest.mark.parametrize("ncell", [5, 8, 12])
def test_pair_list_of_three_edges(ncell):
    s = systems.lj_fluid(ncell=ncell, seed=3, jitter_star=0.1)
    ens, pos, box = _three_edges(s)
    rl = s.config.cutoff + s.config.cut_buffer
    i, j = np.triu_indices(s.n_atoms, 1)
    d = pos[j] - pos[i]
    d -= box * np.round(d / box)
    take = (d ** 2).sum(1) < rl * rl
    want = np.stack([i[take], j[take]], 1)
    got = ens.pairs()
    assert np.array_equal(got[np.lexsort((got[:, 1], got[:, 0]))], want)
    ens.close()


# flexible water without cells and with 3 x 3 x 4 at rest, without and with
# 4 x 4 x 5 under shear
@pytest.mark.parametrize("rate,nmol", [(0.0, 343), (0.0, 1400), (5.0, 343), (5.0, 3000)])
def test_water_of_three_edges(rate, nmol):
    s = systems.spce_flexible(nmol=nmol, seed=2, strain_rate=rate)
    ens, _, box = _three_edges(s)
    nh = engine.NHIntegrator(ens)
    nh.start()
    nh.run(40)
    delta = nh.observables().shear_offset
    pos = ens.state()["pos"]
    ref = oracle.flex_le_forces(s, pos, box, delta)
    # forces and charges as in the cubic box.  The mixed path forms r^2 in FP32
    # here: two roundings a component and three of the sum, 9 of 2^-24, six
    # times that in r^-12
    for precision, tol, tol_vdw in (("fp64", 1e-9, 1e-9), ("mixed", 1e-6, 54 * 2.0 ** -24)):
        ens.set_precision(precision)
        f, e, w = ens.compute_forces()
        assert ens.ewald_nk() == ref["nk"]
        assert rms_rel(f, ref["force"]) < tol
        for idx, key in ((L.E_VDW, "vdw"), (L.E_REAL, "real"), (L.E_LONG, "long"), (L.E_MOLCORRECT, "intra")):
            assert abs(e[idx] - ref[key]) < (tol_vdw if key == "vdw" else tol) * abs(ref[key]) + 1e-9, key
        assert np.max(np.abs(w - ref["virial"])) < 10 * tol * np.abs(ref["virial"]).max()
    ens.close()


# multipole columns against one FP64 sine and cosine per (site, k)
@pytest.mark.parametrize("kmax", [3, 8, 14])
def test_multipole_columns_of_three_edges(kmax):
    s = systems.polarizable_water(nmol=343, cutoff=0.9, switch=0.8, kmax=kmax, seed=7)
    ens, _, _ = _three_edges(s)
    ens.set_solver(tol=1e-13, max_iter=1000)
    terms = L.TERM_MP_SHORT | L.TERM_MP_LONG | L.TERM_IND_SHORT | L.TERM_IND_LONG
    ens.set_reference_forms(True)
    ref = [ens.compute_forces(t) for t in (terms, L.TERM_MP_LONG)]
    ens.set_reference_forms(False)
    for precision, tol in (("fp64", 1e-10), ("mixed", 1e-6)):
        ens.set_precision(precision)
        for (f, e, w), t in zip(ref, (terms, L.TERM_MP_LONG)):
            fm, em, wm = ens.compute_forces(t)
            assert rms_rel(fm, f) < tol
            for q in (L.E_LONG, L.E_POL_LONG):
                assert abs(em[q] - e[q]) <= tol * abs(e[q])
            assert np.abs(wm - w).max() < tol * np.abs(w).max()
    ens.close()


def _by_site(s):
    """s with every molecule's first site first, then every second one, ...:
    (the system, old index of each new site)."""
    ns = s.n_atoms // s.n_mols
    old = np.arange(s.n_atoms).reshape(s.n_mols, ns).T.reshape(-1)
    new = np.argsort(old)
    bonds, angles = s.bonds.copy(), s.angles.copy()
    bonds[:, :2], angles[:, :3] = new[bonds[:, :2]], new[angles[:, :3]]
    return s.replace(pos=s.pos[old], atom_type=s.atom_type[old], mol_id=s.mol_id[old], bonds=bonds,
                     angles=angles), old


# rigid water (SHAKE), flexible water (leap-frog and chain under shear): the
# trajectory does not depend on the order of the sites.  Forces differ by the
# order of their FP64 sums and 2^-32, over some steps by far less than 1e-9
@pytest.mark.parametrize("kind", ["shake", "free", "chain"])
def test_trajectory_of_sites_by_kind(kind):
    if kind == "shake":
        s = systems.spce_water(nmol=343, box=2.19, cutoff=0.9, kmax=6, seed=4)
    else:
        s = systems.spce_flexible(nmol=343, seed=4, strain_rate=5.0 if kind == "chain" else 0.0)
    out = []
    for t, old in ((s, np.arange(s.n_atoms)), _by_site(s)):
        v = engine.init_velocity(s)
        ens = engine.GpuEnsemble(t, velocities=v[old])
        lf = (engine.NHIntegrator if kind == "chain" else engine.LFIntegrator)(ens)
        lf.start()
        lf.run(30)
        st, o = ens.state(), lf.observables()
        p = ens.pairs()
        p = np.sort(old[p], axis=1)
        out.append((st["pos"][np.argsort(old)], st["vel"][np.argsort(old)],
                    np.array([o.e_potential, o.ke_atom, o.ke_mol, *o.atom_pressure, *o.mol_pressure]),
                    p[np.lexsort((p[:, 1], p[:, 0]))]))
        ens.close()
    a, b = out
    assert np.abs(a[0] - b[0]).max() < 1e-9
    assert np.abs(a[1] - b[1]).max() < 1e-9 * np.abs(a[1]).max()
    assert np.allclose(a[2], b[2], rtol=1e-9, atol=1e-9 * np.abs(a[2]).max())
    assert np.array_equal(a[3], b[3])


def test_step_of_mixed_molecule_lengths():
    """Molecules of three sites and of one in one system: the list against all
    pairs, one free step against the leap-frog formulas."""
    s = systems.spce_flexible(nmol=343, seed=4)
    split = 3 * 300   # the last 43 waters as single sites
    s.mol_id = s.mol_id.copy()
    s.mol_id[split:] = 300 + np.arange(s.n_atoms - split)
    s.bonds, s.angles = s.bonds[(s.bonds[:, 0] < split)], s.angles[s.angles[:, 0] < split]
    s.mol_type_names = [("WAT", 3), ("ION", 1)]
    s.mol_type = np.array([0] * 300 + [1] * (s.n_atoms - split), np.int32)
    s.config.thermostat = "none"
    m, box = s.masses()[:, None], s.box[0]
    v = np.random.default_rng(1).normal(size=s.pos.shape)
    v -= (m * v).sum(0) / m.sum()
    ens = engine.GpuEnsemble(s, velocities=v)
    i, j = np.triu_indices(s.n_atoms, 1)
    d = s.pos[j] - s.pos[i]
    d -= box * np.round(d / box)
    take = (d ** 2).sum(1) < (s.config.cutoff + s.config.cut_buffer) ** 2
    ex = {(a, b) for a, l in enumerate(s.exclusion_table()) for b in l}
    want = [(a, b) for a, b in zip(i[take], j[take]) if (a, b) not in ex]
    got = ens.pairs()
    assert np.array_equal(got[np.lexsort((got[:, 1], got[:, 0]))], want)
    f, _, _ = ens.compute_forces()
    lf = engine.LFIntegrator(ens)
    lf.start()
    lf.run(1)
    st, o, dt = ens.state(), lf.observables(), s.config.timestep
    vm, vp = v - 0.5 * dt * f / m, v + 0.5 * dt * f / m
    pos = s.pos + dt * vp
    com = np.stack([np.bincount(s.mol_id, (m * pos)[:, x]) for x in range(3)], 1) / np.bincount(s.mol_id, m[:, 0])[:, None]
    pos = pos - (box * np.round(com / box))[s.mol_id]
    assert np.abs(st["pos"] - pos).max() < 1e-12
    assert np.abs(st["vtminus"] - vp).max() < 1e-11
    assert abs(o.ke_atom - 0.5 * (m * v * v).sum()) < 1e-10 * o.ke_atom
    p = np.stack([np.bincount(s.mol_id, (m * v)[:, x]) for x in range(3)], 1)
    assert abs(o.ke_mol - 0.5 * (p ** 2 / np.bincount(s.mol_id, m[:, 0])[:, None]).sum()) < 1e-10 * o.ke_mol
    ens.close()
