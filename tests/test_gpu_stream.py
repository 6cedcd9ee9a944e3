"""The device generator across its refills: runs of one move, of a few, across the
624-word blocks and the 256-move batches, on one seed, against the same moves on a
recorded mt19937 stream (the same draws: equal energies and positions)."""
import numpy as np
import pytest

from plum_gb300 import systems


@pytest.mark.gpu
@pytest.mark.parametrize("form", [0, 1])
def test_device_stream_equals_recorded(tmp_path, built, form):
    import plum_gb300 as pg
    spec = systems.BulkSpec(n_chain=4, chain_len=12, n_ion=48, box=16.0)
    systems.write_bulk(str(tmp_path), spec, seed=3)
    a, b = pg.System(str(tmp_path), form=form), pg.System(str(tmp_path), form=form)
    a.seed(77)
    runs = (1, 1, 7, 2, 64, 255, 256, 257, 3, 600)
    for n in runs:
        a.run(n)
    b.run_moves(built.mt19937(77, 400000), sum(runs))
    np.testing.assert_array_equal(a.positions(), b.positions())
    np.testing.assert_array_equal(a.energies(), b.energies())


@pytest.mark.gpu
def test_dropped_words_are_skipped(tmp_path):
    """A recorded stream drops the generator's unread words up to the end of a full
    buffer, whatever part of it had been made: 4 M words here, so that the moves after
    it are those of a generator that starts there."""
    import plum_gb300 as pg
    spec = systems.BulkSpec(n_chain=4, chain_len=12, n_ion=48, box=16.0)
    systems.write_bulk(str(tmp_path), spec, seed=3)
    a, b = pg.System(str(tmp_path)), pg.System(str(tmp_path))
    words = np.random.RandomState(99).randint(0, 2**32, (1 << 22) + 400000, dtype=np.uint32)
    a.seed(99)
    a.run(40)
    x = a.positions()
    a.run_moves(words[:20000], 5)
    a.set_positions(x)
    a.total_energy()
    a.run(300)
    b.set_positions(x)
    b.total_energy()
    b.run_moves(words[1 << 22:], 300)
    np.testing.assert_array_equal(a.positions(), b.positions())
