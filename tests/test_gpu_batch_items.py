"""The batched energy change over its item sizes (k items of 32 to 512 units, pair
items of 1,024 to 32,768 pairs, each register budget) and real-space rules (one
image, a second image per axis, a cut-off beyond the box): after 48 moves the
running energies equal a from-scratch FP64 recompute within 2e-5 of the energy
change's scale per move (tests/test_gpu_fp32.py), and the tunes agree."""
import numpy as np
import pytest

from plum_gb300 import systems

BOX, MOVES = 16.0, 48


@pytest.mark.gpu
@pytest.mark.parametrize("rule", ["half", "auto", "beyond"])
def test_running_energies_across_tunes(tmp_path, rule):
    import plum_gb300 as pg
    over = {"half": dict(real_cutoff=0.5 * BOX, kmax=5, kcut2=-1.0), "auto": {},
            "beyond": dict(real_cutoff=1.125 * BOX, kmax=4, kcut2=-1.0)}[rule]
    spec = systems.BulkSpec(n_chain=3, chain_len=41, n_ion=123, box=BOX, **over)
    systems.write_bulk(str(tmp_path), spec, seed=6)
    first = None
    for tune in ((1024, 64, 0, 2), (4096, 128, 608, 4), (2048, 256, 304, 3), (32768, 1024, 64, 3)):
        b = pg.Batch([str(tmp_path)] * 3)
        b.seed(np.arange(3, dtype=np.uint32) + 9)
        b.set_tune(*tune)
        b.run(MOVES)
        got = b.energies()
        for r in range(3):
            want = b.replica(r).total_energy()[:4]
            scale = max(1.0, np.abs(want).max())
            assert np.abs(got[r] - want).max() <= MOVES * 2e-5 * scale, (tune, r, got[r], want)
        if first is None:
            first = got
        np.testing.assert_allclose(got, first, rtol=0, atol=MOVES * 2e-5 * max(1.0, np.abs(first).max()))
        b.close()
