"""Words that a recorded stream drops, at every stage of the device generator's buffer:
the moves after it are those of a generator that has passed the end of a full buffer of
4 x 256 x (16 + 12 x longest chain) words, refilled whenever fewer than 256 moves' worth
are left before a batch of 256. Most moves pivot a long chain, some 1,250 words a
move on average, so a few batches reach each stage: the first fill, the second (which the
full buffer's end cuts short), the last words of the full buffer, its refill. (Those
pivots are rejected; the ions' moves show which words were drawn.)"""
import numpy as np
import pytest

from plum_gb300 import systems

LEN, SEED = 500, 41
PER_MOVE = 16 + 12 * LEN
FULL = max(4 * 256 * PER_MOVE, 1 << 22)


@pytest.mark.gpu
@pytest.mark.parametrize("runs", [(1,), (300,), (1800,), (3500,), (5100,), (1, 7, 300, 2100, 3),
                                  (1000, 1000, 1000, 5)])
def test_dropped_words_at_every_stage(tmp_path, runs):
    import plum_gb300 as pg
    spec = systems.BulkSpec(n_chain=1, chain_len=LEN, n_ion=40, box=40.0, real_cutoff=20.0, kmax=2,
                            kcut2=-1.0, move_prob=(0.3, 0.0, 0.7, 0.0, 0.0))
    systems.write_bulk(str(tmp_path), spec, seed=3)
    words = np.random.RandomState(SEED).randint(0, 2**32, 3 * FULL, dtype=np.uint32)
    a, b = pg.System(str(tmp_path)), pg.System(str(tmp_path))
    a.seed(SEED)
    used = left = 0
    for n in runs:
        a.run(n)
        while n:  # the same moves on the recorded words, which tells how many they take
            if left < 256 * PER_MOVE:
                left = FULL
            k = min(n, 256)
            took = b.run_moves(words[used:used + 256 * PER_MOVE], k, logs=False)[0]
            used, left, n = used + took, left - took, n - k
    x = a.positions()
    np.testing.assert_array_equal(x, b.positions())
    a.run_moves(words[:40000], 5)
    for s in (a, b):
        s.set_positions(x)
    assert a.run(40) > 0
    b.run_moves(words[used + left:used + left + 256 * PER_MOVE], 40)
    np.testing.assert_array_equal(a.positions(), b.positions())
    np.testing.assert_array_equal(a.energies(), b.energies())
