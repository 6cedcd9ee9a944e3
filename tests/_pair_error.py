"""How far an energy change of the precision form may be off, for the tests that compare
one move's with the difference of two from-scratch FP64 energies.

Per pair of a moved bead, at its old and its new place. r^2 carries some eight roundings
of 2^-24 (differences, squares, sums, scales), so a term f(r^2) is off by 5e-7 |r^2 f'|;
a term's own evaluation and the sums (FP32 within a block: some forty adds) by 1e-6 |f|;
and positions are fixed point, 2^-32 of the box per bead and axis, so r by at most
2^-30 L. LJ: sigma = eps = 1. The 2e-5 of the energy change covers the reciprocal part,
as in tests/test_gpu_fp32.py."""
import numpy as np


def allowance(info, q, old, new, moved, delta, lj_cut=2.5):
    """old, new: positions; moved: bead indices; delta: the energy change's terms."""
    import torch
    tol = 2e-5 * max(1.0, float(np.abs(delta).max()))
    box = torch.tensor(list(info.ewald_box), dtype=torch.float64, device="cuda")
    quant = float(box.max()) * 2.0 ** -30
    n = torch.tensor([-1.0, 0.0, 1.0], dtype=torch.float64, device="cuda")
    images = torch.cartesian_prod(n, n, n)
    qt = torch.as_tensor(np.asarray(q, np.float64), device="cuda")
    idx = torch.as_tensor(np.asarray(moved), device="cuda")
    qq = (qt[None] * qt[idx][:, None]).abs() * info.lB
    for xyz in (old, new):
        x = torch.as_tensor(np.asarray(xyz), device="cuda")
        d = x[None] - x[idx][:, None]
        d = d - box * torch.round(d / box)
        r = d.norm(dim=2)
        near = (r > 0) & (r < lj_cut)
        s6 = torch.where(near, r, torch.full_like(r, 1e9)) ** -6
        slope = 24 * (2 * s6 * s6 + s6)  # r |U'| and more
        tol += float((5e-7 * slope / 2 + 1e-6 * 4 * (s6 * s6 + s6)).sum())
        tol += quant * float((slope / r.clamp(min=1e-3)).sum())
        r = (d[:, :, None] + images * box).norm(dim=3)  # the image cells
        u = info.alpha * r * r
        on = (r > 0) & (r <= info.real_cutoff)
        r = r.clamp(min=1e-3)
        t = torch.where(on, qq[:, :, None] * torch.erfc(u.sqrt()) / r, torch.zeros_like(r))
        tol += float((t * (5e-7 * (u + 1) + 1e-6 + quant * (2 * u + 1) / r)).sum())
    return tol
