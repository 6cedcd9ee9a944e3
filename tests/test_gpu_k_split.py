"""The batched energy change's reciprocal part with k items of 32, 64 and 256 units, that is
eight, four and one threads a unit: how a unit's beads are split over threads must not
show in its error (against from-scratch FP64 energies, over some 600 accepted moves of the
same replicas; 1.5 times the one-thread error is allowed for the other order of the sums).
A chain in bulk, and a slab, whose sums over the moved beads are large."""
import numpy as np
import pytest

from plum_gb300 import systems


def errors(path, k_tile, replicas=16, steps=80):
    import plum_gb300 as pg
    b = pg.Batch([path] * replicas)
    b.seed(np.arange(replicas, dtype=np.uint32) + 9)
    b.set_tune(4096, k_tile, 608, 3)
    out = []
    for _ in range(steps):
        e0 = [b.replica(r).total_energy().copy() for r in range(replicas)]
        b.run(1)
        got = b.energies().copy()
        for r in range(replicas):
            t = b.replica(r).total_energy()
            # an energy change has the reference's dipole term, from the current z
            want = t[1] - (t[7] - e0[r][7])
            if 1e-9 < np.abs(t[:4] - e0[r][:4]).max() < 50:
                out.append(got[r][1] - want)
    b.close()
    assert len(out) >= 300
    return float(np.sqrt(np.mean(np.square(out))))


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["bulk", "slab"])
def test_error_does_not_depend_on_the_split(tmp_path, kind):
    if kind == "slab":
        spec = systems.BrushSpec(n_graft=16, chain_len=30, lxy=32.0, height=36.0, n_sites=12,
                                 charge_frac=0.7)
        systems.write_brush(str(tmp_path), spec, seed=6, beta=0.05)
    else:
        spec = systems.BulkSpec(n_chain=3, chain_len=41, n_ion=123, box=16.0)
        systems.write_bulk(str(tmp_path), spec, seed=6, beta=0.05)
    one = errors(str(tmp_path), 1024)
    for k_tile in (64, 128):
        e = errors(str(tmp_path), k_tile)
        assert e <= 1.5 * one, (k_tile, e, one)
