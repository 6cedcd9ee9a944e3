"""Coordinates that are not finite: the kernels hold positions as integer fractions of
the box, which have no NaN, and the energies they enter are NaN all the same, as FP64
positions make them in the reference. A trial move's energy change (both forms), a
stored frame's energy and structure factor, a growth step's trial energies and the
slit pressure; and what comes after, with finite coordinates again, is unchanged."""
import os

import numpy as np
import pytest

from _cases import GOLDEN
from plum_gb300 import systems

NAN, INF = float("nan"), float("inf")
HALF = dict(real_cutoff=7.0, kmax=4, kcut2=-1.0)


def bulk(tmp_path, rule):
    spec = systems.BulkSpec(n_chain=2, chain_len=9, n_ion=18, box=14.0,
                            **(HALF if rule == "half" else {}))
    systems.write_bulk(str(tmp_path), spec, seed=2)
    return str(tmp_path)


@pytest.mark.gpu
@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("system", ["half", "auto", "slab_lj"])
def test_energy_difference_is_nan(tmp_path, form, system):
    import plum_gb300 as pg
    slab = system.startswith("slab")
    s = pg.System(os.path.join(GOLDEN, system) if slab else bulk(tmp_path, system), form=form)
    s.total_energy()
    ms, _, _ = s.topology()
    x0, e0 = s.positions().copy(), s.energies().copy()
    sizes = np.diff(ms)
    chain, ion = int(np.argmax(sizes)), int(len(sizes) - 1)
    assert sizes[chain] > 1 and sizes[ion] == 1

    def change(mol, bead=0, axis=0, to=None):
        n = sizes[mol]
        t = x0[ms[mol]:ms[mol + 1]] + 0.01
        if to is not None:
            t[bead, axis] = to
        got = s.energy_difference(mol, t, np.ones(n, np.int32))
        s.finalize(False)
        return got

    good = [change(ion), change(chain)]
    for axis in range(3):
        for to in (NAN, INF, -INF):
            if slab and axis == 2 and np.isinf(to):
                continue  # past the wall: the overlap value, before any pair
            assert np.isnan(change(ion, 0, axis, to)[0]), (axis, to)
            assert np.isnan(change(chain, sizes[chain] - 1, axis, to)[0]), (axis, to)
    np.testing.assert_array_equal(good, [change(ion), change(chain)])
    np.testing.assert_array_equal(e0, s.energies())
    np.testing.assert_array_equal(x0, s.positions())
    s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("system", ["half", "auto", "slab_lj"])
def test_stored_frame_is_nan(tmp_path, form, system):
    import plum_gb300 as pg
    slab = system.startswith("slab")
    s = pg.System(os.path.join(GOLDEN, system) if slab else bulk(tmp_path, system), form=form)
    want = s.total_energy().copy()
    x0 = s.positions().copy()
    for axis in (0, 1) if slab else (0, 1, 2):
        for to in (NAN, INF):
            x = x0.copy()
            x[len(x) // 2, axis] = to
            s.set_positions(x)
            assert np.isnan(s.total_energy()[1]), (axis, to)
            assert np.isnan(s.structure_factor()[0]).any(), (axis, to)
    s.set_positions(x0)
    np.testing.assert_array_equal(want, s.total_energy())
    s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("charge", [0.0, -1.0])
def test_trial_site_is_nan(tmp_path, charge, pinned):
    import plum_gb300 as pg
    spec = systems.MuVTSpec(box=14.0, n_chain=3, chain_len=9, bead_charge=charge, n_salt=20)
    over = HALF if pinned else dict(real_cutoff=11.0)
    systems.write_muvt(str(tmp_path), spec, seed=3, **over)
    s = pg.System(str(tmp_path))
    rng = np.random.default_rng(4)
    T, cl = 33, 3
    chain = rng.uniform(0, 14, (cl, 3))
    ci = rng.uniform(0, 14, (cl, 3)) if charge else None
    b1 = rng.uniform(0, 14, (T, 3))
    b2 = rng.uniform(0, 14, (T, 3)) if charge else None
    want = s.cbmc_trials(b1, b2, chain, ci)
    free = want < 1e8
    assert free.sum() > T // 2
    for axis in range(3):
        for to in (NAN, INF):
            at = int(np.flatnonzero(free)[axis])
            for which in (b1, b2) if charge else (b1,):
                old = which[at, axis]
                which[at, axis] = to
                got = s.cbmc_trials(b1, b2, chain, ci)
                which[at, axis] = old
                assert np.isnan(got[at]), (axis, to)
                others = np.arange(T) != at
                np.testing.assert_array_equal(got[others], want[others])
            bad = chain.copy()
            bad[1, axis] = to
            assert np.isnan(s.cbmc_trials(b1, b2, bad, ci)[free]).all(), (axis, to)
    np.testing.assert_array_equal(want, s.cbmc_trials(b1, b2, chain, ci))
    s.close()


@pytest.mark.gpu
def test_slit_pressure_is_nan():
    import plum_gb300 as pg
    s = pg.System(os.path.join(GOLDEN, "slab_charged_sites"))
    want = s.pressure_slit().copy()
    _, q, _ = s.topology()
    at = int(np.flatnonzero(q)[-1])
    x0 = s.positions().copy()
    for axis in range(2):
        x = x0.copy()
        x[at, axis] = NAN
        s.set_positions(x)
        assert np.isnan(s.pressure_slit()[3:]).any(), axis
    s.set_positions(x0)
    np.testing.assert_array_equal(want, s.pressure_slit())
    s.close()
