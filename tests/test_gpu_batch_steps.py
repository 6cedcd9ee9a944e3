"""The batched energy change, move by move: the running energies after one accepted move,
from a from-scratch FP64 energy before it, against another one after it, within what
tests/_pair_error.py derives for the beads that moved. Work items of different sizes, each
register budget, both pair loops; one image, a second one per axis, a cut-off beyond the
box, unequal edges (one image on each axis; on one beside axes with two; images of two
axes at once), a slab. Replicas are
warm (beta = 0.05), so that moves of every kind are accepted."""
import numpy as np
import pytest

from _pair_error import allowance
from plum_gb300 import systems

BOX = 16.0


def make(path, rule, seed):
    if rule == "slab":
        spec = systems.BrushSpec(n_graft=4, chain_len=21, lxy=BOX, height=18.0, n_sites=3,
                                 charge_frac=0.7)
        systems.write_brush(path, spec, seed=seed, beta=0.05)
        return
    over = {"half": dict(real_cutoff=0.5 * BOX, kmax=5, kcut2=-1.0), "auto": {},
            "beyond": dict(real_cutoff=1.125 * BOX, kmax=4, kcut2=-1.0),
            "edges": dict(real_cutoff=10.0, kmax=5, kcut2=-1.0),
            "edges_two": dict(real_cutoff=13.0, kmax=5, kcut2=-1.0),
            "edges_half": dict(real_cutoff=8.0, kmax=5, kcut2=-1.0)}[rule]
    spec = systems.BulkSpec(n_chain=3, chain_len=41, n_ion=123, box=BOX)
    systems.write_bulk(path, spec, seed=seed, beta=0.05, **over)
    if rule.startswith("edges"):
        systems.write_top(path + "/input_top.dat", 246, 126, (BOX, 1.15 * BOX, 1.5 * BOX))


@pytest.mark.gpu
@pytest.mark.parametrize("tune", [(1024, 64, 0, 2), (4096, 128, 608, 4), (32768, 1024, 64, 3)])
@pytest.mark.parametrize("rule", ["half", "auto", "beyond", "edges", "edges_two", "edges_half",
                                  "slab"])
def test_each_accepted_move(tmp_path, rule, tune):
    import plum_gb300 as pg
    make(str(tmp_path), rule, 6)
    b = pg.Batch([str(tmp_path)] * 3)
    b.seed(np.arange(3, dtype=np.uint32) + 9)
    b.set_tune(*tune)
    q = b.replica(0).topology()[1]
    n_chain = 0
    kinds = set()
    loops = (1, 0) if b.real_term() else (0,)
    for step in range(40):
        b.set_real_term(loops[step % len(loops)])
        old = [b.replica(r).positions().copy() for r in range(3)]
        e0 = [b.replica(r).total_energy().copy() for r in range(3)]
        b.run(1)
        got = b.energies().copy()
        for r in range(3):
            s = b.replica(r)
            new = s.positions().copy()
            moved = np.flatnonzero((new != old[r]).any(axis=1))
            t = s.total_energy()
            want = t[:4].copy()
            # an energy change has the reference's dipole term, from the current z
            want[1] -= t[7] - e0[r][7]
            tol = 1e-9 * max(1.0, np.abs(e0[r][:4]).max(), np.abs(want).max())
            if len(moved):
                n_chain += len(moved) > 1
                kinds.add(min(len(moved), 2))
                tol += allowance(s.info, q, old[r], new, moved, want - e0[r][:4])
            assert np.abs(got[r] - want).max() <= tol, (step, r, got[r] - want, tol)
    assert n_chain >= 8 and kinds == {1, 2}
    b.close()
