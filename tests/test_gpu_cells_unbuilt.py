"""The descriptor's cell lists of a batch without a surrogate: never built, so an accepted
move must not follow keys that hold whatever the memory held before. Device memory is
filled with other numbers and given back first; the lists stay empty and invalid, the
moves are those of two step chains, and lists built for a surrogate later on work."""
import numpy as np
import pytest

from plum_gb300 import systems


@pytest.mark.gpu
def test_moves_leave_unbuilt_lists_alone(tmp_path):
    import torch
    import plum_gb300 as pg
    spec = systems.BulkSpec(n_chain=6, chain_len=24, n_ion=144, box=24.0, kmax=4, kcut2=-1.0,
                            real_cutoff=12.0)
    systems.write_bulk(str(tmp_path), spec, seed=8)
    fill = torch.randint(-2**31, 2**31 - 1, (1 << 28,), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    del fill
    torch.cuda.empty_cache()
    end = []
    for groups in (1, 2):
        b = pg.Batch([str(tmp_path)] * 4)
        b.seed(np.arange(4, dtype=np.uint32) + 21)
        b.set_groups(groups)
        assert b.run(300) > 0
        with_lists, valid, most, _ = b.cell_stats()
        assert (with_lists, valid, most) == (4, 0, 0)
        end.append([b.replica(r).positions().copy() for r in range(4)])
        b.set_cell_cap(64)  # lists in new memory
        assert b.run(50) > 0
        assert b.cell_stats()[1:3] == (0, 0)
        b.set_surrogate(pg.Surrogate(seed=3))
        b.run(20)
        with_lists, valid, most, cap = b.cell_stats()
        assert with_lists == 4 and valid == 4 and 0 <= most <= cap
        b.close()
    np.testing.assert_array_equal(end[0], end[1])
