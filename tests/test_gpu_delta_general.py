"""The general pair loops of the energy-difference kernels (k_delta64<0>, k_delta32<0>:
slabs, hard spheres, r_c beyond the box, unequal edges in FP64), and the precision form's
second image per axis with unequal edges, where their splits over threads and phase-table
chunks change: one moved bead, a few, a chunk of 32 or 64 beads and one more, several.
Against the difference of two from-scratch energies (other kernels, FP64).

Tolerances: 1e-9 of the larger total in FP64 (tests/test_gpu_delta_sizes.py), and what
tests/_pair_error.py derives in the precision form."""
import numpy as np
import pytest

from _pair_error import allowance
from plum_gb300 import systems

BOX = 20.0
HALF = dict(real_cutoff=0.5 * BOX, kmax=5, kcut2=-1.0)


def make(path, kind, length):
    """(molecule to move)"""
    if kind == "slab":
        spec = systems.BrushSpec(n_graft=1, chain_len=length, lxy=BOX, height=24.0, n_sites=3,
                                 charge_frac=0.8)
        systems.write_brush(path, spec, seed=length)
        return 2 * spec.n_sites
    over, top = {}, None
    if kind == "hard":
        over = dict(HALF, pair_kind="HardSphere", hs_radii=(("P", 0.3), ("C", 0.3)))
    elif kind == "beyond":
        over = dict(real_cutoff=1.12 * BOX, kmax=4, kcut2=-1.0)
    else:  # a second image on the two short axes; on all of them, and on two at once
        over = dict(real_cutoff=13.0 if kind == "edges" else 18.0, kmax=5, kcut2=-1.0)
        top = (BOX, 1.25 * BOX, 1.5 * BOX)
    spec = systems.BulkSpec(n_chain=1, chain_len=length, n_ion=200, box=BOX)
    systems.write_bulk(path, spec, seed=length, **over)
    if top:
        systems.write_top(path + "/input_top.dat", length + 200, 201, top)
    return 0


def terms(s):
    """The energy's terms without the dipole's: an energy change has the reference's, from
    the current z."""
    t = s.total_energy().copy()
    t[1] -= t[7]
    return t[:4]


@pytest.mark.gpu
@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("kind", ["slab", "hard", "beyond", "edges", "edges_two"])
@pytest.mark.parametrize("length", [1, 3, 32, 33, 65, 130])
def test_energy_difference_of_the_general_loops(tmp_path, form, kind, length):
    import plum_gb300 as pg
    mol = make(str(tmp_path), kind, length)
    s = pg.System(str(tmp_path), form=form)
    ms, q, _ = s.topology()
    assert ms[mol + 1] - ms[mol] == length
    rng = np.random.default_rng(length)
    x0 = s.positions().copy()
    e0 = terms(s)
    assert np.abs(e0).max() < 1e8  # no overlap to start from
    for lo in sorted({0, length // 3}):
        trial = x0[ms[mol]:ms[mol + 1]].copy()
        trial[lo:] += rng.normal(0, 0.02, 3) + rng.normal(0, 0.01, (length - lo, 3))
        moved = np.zeros(length, np.int32)
        moved[lo:] = 1
        got = s.energy_difference(mol, trial, moved)[0]
        s.finalize(False)
        x1 = x0.copy()
        x1[ms[mol]:ms[mol + 1]] = trial
        s.set_positions(x1)
        e1 = terms(s)
        s.set_positions(x0)
        s.total_energy()
        want = float((e1 - e0).sum())
        tol = 1e-9 * max(1.0, np.abs(e0).max(), np.abs(e1).max())
        if form:
            tol += allowance(s.info, q, x0, x1, ms[mol] + np.arange(lo, length), e1 - e0)
        assert abs(got - want) <= tol, (lo, got, want, tol)
    s.close()
