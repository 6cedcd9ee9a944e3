"""Slabs whose Ewald box is not padded: no dipole correction, or no Ewald term at all. z is
not wrapped, so beads near opposite walls are a gap apart for LJ, and their images along z
count in the real-space sum even with r_c below half of every box length. Totals of the
plain form against the CPU restatement (1e-10), energy changes of both forms against the
difference of two totals (1e-9 of them; tests/_pair_error.py in the precision form), the
batch's accepted moves."""
import numpy as np
import pytest

from _pair_error import allowance
from plum_gb300 import systems

KINDS = {"ewald": dict(dipole=False, real_cutoff=5.0, kmax=4, kcut2=-1.0),
         "ewald_auto": dict(dipole=False), "lj": dict(dipole=False, use_ewald=False)}


def make(path, kind, **over):
    """Chains grafted on one wall, ions near both: a gap of 11, most of it within r_c."""
    spec = systems.BrushSpec(n_graft=5, chain_len=14, lxy=12.0, height=11.0, n_sites=3,
                             charge_frac=0.9)
    systems.write_brush(path, spec, seed=3, **dict(KINDS[kind], **over))


def frames(x, ms, n, seed):
    rng = np.random.default_rng(seed)
    for _ in range(n):
        m = int(rng.integers(6, len(ms) - 1))  # past the wall sites
        a, b = ms[m], ms[m + 1]
        y = x.copy()
        y[a:b] += rng.normal(0, 0.05, 3) * [1, 1, 0.2] + rng.normal(0, 0.01, (b - a, 3))
        if y[a:b, 2].min() > 0.5 and y[a:b, 2].max() < 10.5:
            yield m, y


@pytest.mark.gpu
@pytest.mark.parametrize("kind", sorted(KINDS))
def test_plain_totals_match_the_restatement(tmp_path, built, kind):
    import plum_gb300 as pg
    make(str(tmp_path), kind)
    s, o = pg.System(str(tmp_path)), built.Oracle(str(tmp_path))
    x0 = s.positions().copy()
    for _, x in frames(x0, s.topology()[0], 6, 1):
        s.set_positions(x)
        o.set_coords(x)
        got, want = s.total_energy()[:4], o.total_energy()[:4]
        for a, b in zip(got, want):
            assert abs(a - b) <= 1e-10 * max(1.0, abs(b)), (got, want)
    s.close()
    o.close()


@pytest.mark.gpu
@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("kind", sorted(KINDS))
def test_energy_changes(tmp_path, kind, form):
    import plum_gb300 as pg
    make(str(tmp_path), kind)
    s = pg.System(str(tmp_path), form=form)
    ms, q, _ = s.topology()
    x0 = s.positions().copy()
    e0 = s.total_energy()[:4].copy()
    for m, x in frames(x0, ms, 24, 2):
        a, b = ms[m], ms[m + 1]
        got = s.energy_difference(m, x[a:b], np.ones(b - a, np.int32))[0]
        s.finalize(False)
        s.set_positions(x)
        e1 = s.total_energy()[:4].copy()
        s.set_positions(x0)
        s.total_energy()
        tol = 1e-9 * max(1.0, np.abs(e0).max(), np.abs(e1).max())
        if form:
            tol += allowance(s.info, q if kind != "lj" else 0 * q, x0, x, np.arange(a, b), e1 - e0)
        assert abs(got - float((e1 - e0).sum())) <= tol, (m, got, (e1 - e0).sum(), tol)
    s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("kind", sorted(KINDS))
def test_batch_moves(tmp_path, kind):
    import plum_gb300 as pg
    make(str(tmp_path), kind, beta=0.05)
    b = pg.Batch([str(tmp_path)] * 4)
    b.seed(np.arange(4, dtype=np.uint32) + 3)
    q = b.replica(0).topology()[1] * (kind != "lj")
    n = 0
    for _ in range(30):
        old = [b.replica(r).positions().copy() for r in range(4)]
        e0 = [b.replica(r).total_energy()[:4].copy() for r in range(4)]
        b.run(1)
        got = b.energies().copy()
        for r in range(4):
            s = b.replica(r)
            new = s.positions().copy()
            moved = np.flatnonzero((new != old[r]).any(axis=1))
            want = s.total_energy()[:4].copy()
            tol = 1e-9 * max(1.0, np.abs(e0[r]).max(), np.abs(want).max())
            if len(moved):
                n += 1
                tol += allowance(s.info, q, old[r], new, moved, want - e0[r])
            assert np.abs(got[r] - want).max() <= tol, (r, got[r] - want, tol)
    assert n >= 20
    b.close()
