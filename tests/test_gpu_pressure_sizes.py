"""The slit-pressure kernels at the edges of their blocks: one site per wall,
one more than a chunk of staged sites, more than two chunks; bead counts below
and just above one tile of 256 (charged sites, so that no column is zero),
against the CPU restatement at the tolerance of tests/test_slit_pressure.py."""
import numpy as np
import pytest

from plum_gb300 import systems


@pytest.mark.gpu
@pytest.mark.parametrize("n_graft,chain_len,n_sites", [(2, 5, 1), (5, 27, 33), (9, 21, 65)])
def test_pressure_at_block_edges(built, tmp_path, n_graft, chain_len, n_sites):
    import plum_gb300 as pg
    spec = systems.BrushSpec(n_graft=n_graft, chain_len=chain_len, lxy=16.0, height=31.0,
                             n_sites=n_sites, site_charge=0.5)
    d = str(tmp_path)
    systems.write_brush(d, spec, seed=7 + n_sites)
    o = built.Oracle(d, seed=3)
    want = o.pressure_force_slit()[6:12]
    o.close()
    s = pg.System(d)
    np.testing.assert_allclose(s.pressure_slit(), want, rtol=1e-9, atol=1e-11)
    s.close()
