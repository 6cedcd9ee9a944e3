"""The one-launch FP64 trial kernel at the edges of its chunks (128 trials) and
lists: one trial to two chunks and a bit, no grown bead to more than a warp of
them, a deleted chain, neutral and charged species, r_c = L / 2 (one image) and
the reference's rule at L = 14 (image cells); against the general FP64 kernels,
which plum_cbmc_trials_noalloc runs, at the tolerance of tests/test_zz_no_alloc.py
(1e-10 of max(1, |u|))."""
import ctypes as C

import numpy as np
import pytest

from plum_gb300 import systems


def general(pg, s, b1, b2, chain, ci, did):
    import torch
    d = [None if x is None else torch.as_tensor(np.ascontiguousarray(x, np.float64).ravel(),
                                                device="cuda") for x in (b1, b2, chain, ci)]
    u = torch.zeros(len(b1), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    err = C.create_string_buffer(256)
    f = pg.lib().plum_cbmc_trials_noalloc
    f.argtypes = [C.c_void_p, C.c_int, C.c_void_p, C.c_void_p, C.c_int, C.c_void_p, C.c_void_p,
                  C.c_int, C.c_void_p, C.c_char_p, C.c_int]
    ptr = [C.c_void_p(None if x is None else x.data_ptr()) for x in d]
    rc = f(s.h, len(b1), ptr[0], ptr[1], 0 if chain is None else len(chain), ptr[2], ptr[3], did,
           C.c_void_p(u.data_ptr()), err, 256)
    assert rc == 0, err.value
    return u.cpu().numpy()


@pytest.mark.gpu
@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("charge", [0.0, -1.0])
def test_one_launch_matches_general_kernels(tmp_path, charge, pinned):
    import plum_gb300 as pg
    spec = systems.MuVTSpec(box=14.0, n_chain=3, chain_len=9, bead_charge=charge, n_salt=60)
    over = dict(real_cutoff=7.0, kmax=4, kcut2=-1.0) if pinned else dict(real_cutoff=11.0)
    systems.write_muvt(str(tmp_path), spec, seed=3, **over)
    s = pg.System(str(tmp_path))
    rng = np.random.default_rng(4)
    n_mol = s.n_mol
    last = n_mol - 2 * spec.n_salt - (10 if charge else 1)  # the last chain
    for T, cl, did in ((1, 0, -1), (32, 1, -1), (127, 33, -1), (128, 9, last), (129, 40, -1),
                       (256, 3, -1)):
        chain = rng.uniform(0, 14, (cl, 3)) if cl else None
        ci = rng.uniform(0, 14, (cl, 3)) if cl and charge else None
        b1 = rng.uniform(-3, 17, (T, 3))
        b2 = rng.uniform(-3, 17, (T, 3)) if charge else None
        want = general(pg, s, b1, b2, chain, ci, did)
        got = s.cbmc_trials(b1, b2, chain, ci, did)
        both = (want >= 1e8) & (got >= 1e8)
        tol = 1e-10 * np.maximum(1.0, np.abs(want))
        assert np.all(both | (np.abs(got - want) <= tol)), (T, cl, np.abs(got - want).max())
    s.close()
