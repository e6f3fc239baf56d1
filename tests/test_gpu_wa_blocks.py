"""Nets per thread of the wirelength pass: up to 608 blocks one each, above that
several, by degree class.  On either side every net is counted once: the HPWL total
is the oracle's and the sum of the nets' own values.  (The gradients' accuracy is
tested in test_gpu_parity.py.)"""
import numpy as np
import pytest

from designs import small_synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [120000, 150000, 260000])
def test_wirelength_at_the_block_rule(cells):
    import reda_erplacer_gb300 as R
    from oracle import erp_oracle as O
    d = small_synth(cells, seed=13, macros=2, io=40)
    o = O.Oracle(d, 64, 64, target_density=1.0, start_mode=O.START_DB, density_mode=O.DENSITY_FIXED, reduce_fp64=1)
    g = R.Placement(d, (64, 64), 1.0, start_mode=1)
    try:
        want, got = o.compute_hpwl(60.0), g.compute_hpwl(60.0)
        # per net three FP32 roundings of sums of four coordinates (2^-24 each of the
        # die's size, far above a net's), averaged over 1e5 nets: 1e-6 of the total
        assert abs(got - want) <= 1e-6 * want
        assert abs(float(g.array("NET_HPWL").astype(np.float64).sum()) - got) <= 1e-6 * got
    finally:
        g.close()
        o.close()
