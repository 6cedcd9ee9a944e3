"""How exact the phases of a from-scratch S(k) are: few beads and high orders, so that the
phases' error rules, against long double. A bead's e^{i theta} per axis is good to 2^-53
(its fraction of a turn is carried beyond 64 bits' rounding of w / L, which alone is
2.5e-16), its n-th power to n times that, and three products round once each: the root
mean square over k of |S - S_exact| is at most 2^-53 (|n| + 3) sqrt(sum q^2). Boxes whose
edges have inexact reciprocals, a cubic and a slab's."""
import numpy as np
import pytest

from plum_gb300 import systems

KPI = 3.14159265359  # the reference's constant


@pytest.mark.gpu
@pytest.mark.parametrize("box,slab", [(80.0, False), (16.3, False), (20.0, True)])
def test_structure_factor_of_few_beads(tmp_path, box, slab):
    import plum_gb300 as pg
    if slab:
        spec = systems.BrushSpec(n_graft=6, chain_len=12, lxy=box, height=21.0, n_sites=2, kmax=14,
                                 kcut2=-1.0, real_cutoff=9.0, charge_frac=1.0)
        systems.write_brush(str(tmp_path), spec, seed=4)
    else:
        spec = systems.BulkSpec(n_chain=4, chain_len=16, n_ion=64, box=box, kmax=14, kcut2=-1.0,
                                real_cutoff=0.5 * box)
        systems.write_bulk(str(tmp_path), spec, seed=4)
    s = pg.System(str(tmp_path))
    s.total_energy()
    sk, kn = s.structure_factor()
    q = s.topology()[1].astype(np.longdouble)
    L = np.array(list(s.info.ewald_box), np.longdouble)
    x = s.positions().astype(np.longdouble)
    per = np.array([1, 1, 0 if slab else 1])
    w = x - per * L * np.floor(x / L)
    pick = np.flatnonzero(np.abs(kn).max(axis=1) >= 7)
    pick = np.random.default_rng(0).choice(pick, min(600, len(pick)), replace=False)
    ratio = []
    for k in pick:
        th = 2 * np.longdouble(KPI) * (w @ (kn[k] / L))
        err = np.hypot(sk[k].real - (q * np.cos(th)).sum(), sk[k].imag - (q * np.sin(th)).sum())
        n = np.sqrt(float((kn[k].astype(float) ** 2).sum()))
        ratio.append(float(err) / (2.0 ** -53 * (n + 3) * float(np.sqrt((q * q).sum()))))
    rms = float(np.sqrt(np.mean(np.square(ratio))))
    assert rms <= 1.0, rms
    s.close()
