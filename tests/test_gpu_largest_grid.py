"""Placement on the largest grids that the library takes, where the scatter order counts
more sort tiles than fit a kernel's unasked shared memory (4096 x 4096), and one step
below: the int64 map is the oracle's bit for bit, fresh and after the order was
computed again, and the context steps on."""
import numpy as np
import pytest

from designs import small_synth, spread_positions

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n", [(4096, 2048), (4096, 4096)])
def test_density_on_the_largest_grids(m, n):
    import reda_erplacer_gb300 as R
    from oracle import erp_oracle as O
    d = small_synth(2500, seed=17, macros=1, io=20)
    o = O.Oracle(d, m, n, target_density=1.0, start_mode=O.START_DB, density_mode=O.DENSITY_FIXED, reduce_fp64=1)
    g = R.Placement(d, (m, n), 1.0, start_mode=1)
    try:
        x, y = spread_positions(d, seed=2, frac=0.8)
        o.set_positions(x, y)
        g.set_positions(x, y)
        for again in range(2):
            _, ovo = o.compute_potential(0)
            _, ovg = g.compute_potential(0)
            assert np.array_equal(g.array("DENSITY_I64"), o.get("density_i64"))
            assert abs(ovg - ovo) <= 1e-6 * abs(ovo)
            if again == 0:   # 17 steps: the order is computed from the moved cells
                for _ in range(17):
                    g.step(stats=False)
                assert g.scalars()["iteration"] == 17
                o.set_positions(*g.positions())
    finally:
        g.close()
        o.close()
