"""The autotuner times each of its 4 x 3 x 5 x 3 work-item sizes once (k tiles of 512
and 1,024 vectors are the same kernel), and the other pair loop at the chosen one; the
timed steps are ordinary steps of the replicas, so they end where as many steps of a run
end."""
import numpy as np
import pytest

from _cases import load


@pytest.mark.gpu
def test_each_candidate_is_timed_once():
    import plum_gb300 as pg
    d, _ = load("bulk_small")
    a, b = pg.Batch([d] * 2), pg.Batch([d] * 2)
    for s in (a, b):
        s.seed(np.arange(2, dtype=np.uint32) + 5)
    kt = a.autotune(2)[1]
    assert kt in (128, 256, 512) and b.real_term() == 1
    b.run(2 * (4 * 3 * 5 * 3 + 1))
    for r in range(2):
        np.testing.assert_array_equal(a.replica(r).positions(), b.replica(r).positions())
    a.close()
    b.close()
