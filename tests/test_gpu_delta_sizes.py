"""The energy-difference kernels where their splits change: one moved bead, a few,
the 256 beads staged at a time and one more, two groups, enough pairs for every run
length; one image and image cells; both forms. Against the difference of two
from-scratch energies (other kernels, FP64).

Tolerances. FP64: 1e-9 of the larger total (the difference cancels all but that).
FP32: u carries a relative error of a few 2^-24 and u |dln h/du| is at most some 10 at
the cut-off, so 1e-6 of the sum of the real-space terms' magnitudes, plus the 2e-5 of
the energy change that tests/test_gpu_fp32.py allows for the rest."""
import numpy as np
import pytest

from plum_gb300 import systems

BOX, LB = 30.0, 3.0


def real_terms(xyz, q, idx, rc, alpha):
    import torch
    x = torch.as_tensor(xyz, device="cuda")
    q = torch.as_tensor(q, device="cuda", dtype=torch.float64)
    d = x[None] - x[idx][:, None]
    d -= BOX * torch.round(d / BOX)
    r = d.norm(dim=2)
    t = (q[None] * q[idx][:, None]).abs() * torch.erfc(alpha ** 0.5 * r) / r.clamp(min=1e-9)
    return LB * float(torch.where(r < rc, t, torch.zeros_like(t)).sum())


@pytest.mark.gpu
@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("rule", ["half", "auto"])
@pytest.mark.parametrize("length", [1, 3, 255, 256, 257, 513, 800])
def test_energy_difference_across_splits(tmp_path, form, rule, length):
    import plum_gb300 as pg
    n_ion = 200 if length > 1 else 401
    over = dict(real_cutoff=0.5 * BOX, kmax=5, kcut2=-1.0) if rule == "half" else {}
    spec = systems.BulkSpec(n_chain=1, chain_len=length, n_ion=n_ion, box=BOX, lB=LB, **over)
    systems.write_bulk(str(tmp_path), spec, seed=length)
    s = pg.System(str(tmp_path), form=form)
    _, _, xyz, q = systems.bulk_coordinates(spec, length)
    rc, alpha = (over.get("real_cutoff", 0.7 * BOX)), (spec.alpha_times_L / BOX) ** 2
    rng = np.random.default_rng(length)
    x0 = s.positions().copy()
    e0 = s.total_energy()[:4].copy()
    for lo in sorted({0, length // 3}):
        trial = x0[:length].copy()
        trial[lo:] += rng.normal(0, 0.02, 3) + rng.normal(0, 0.01, (length - lo, 3))
        moved = np.zeros(length, np.int32)
        moved[lo:] = 1
        got = s.energy_difference(0, trial, moved)[0]
        s.finalize(False)
        x1 = x0.copy()
        x1[:length] = trial
        s.set_positions(x1)
        e1 = s.total_energy()[:4].copy()
        s.set_positions(x0)
        s.total_energy()
        want = float((e1 - e0).sum())
        tol = 1e-9 * max(1.0, np.abs(e0).max(), np.abs(e1).max())
        if form:
            idx = np.arange(lo, length)
            tol += 1e-6 * (real_terms(x0, q, idx, rc, alpha) + real_terms(x1, q, idx, rc, alpha))
            tol += 2e-5 * max(1.0, np.abs(e1 - e0).max())
        assert abs(got - want) <= tol, (lo, got, want, tol)
    s.close()
