"""The density scatter's work items: runs of one sort tile's cells, cut at the
item size.  The int64 map is the oracle's, bit for bit, at sizes around the item
bounds, on grids smaller and larger than a tile or a window, with the order fresh
and stale (all cells moved by several bins since it was computed), on both sides
of the size from which the window follows the cells."""
import numpy as np
import pytest

from designs import small_synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells,m,n", [(2, 16, 16), (31, 32, 16), (257, 64, 64), (513, 16, 256), (4097, 64, 128),
                                       (20011, 256, 32), (131071, 256, 256), (131072, 256, 512)])
def test_map_is_the_oracles(cells, m, n):
    import reda_erplacer_gb300 as R
    from oracle import erp_oracle as O
    d = small_synth(cells, seed=cells, macros=1, io=8)
    o = O.Oracle(d, m, n, target_density=1.0, density_mode=O.DENSITY_FIXED, reduce_fp64=1)
    g = R.Placement(d, (m, n), 1.0)
    try:
        k = d.num_movable
        rng = np.random.default_rng(3)
        room_x, room_y = np.maximum(d.die_w - d.w[:k] - 1, 0), np.maximum(d.die_h - d.h[:k] - 1, 0)   # a tiny die has none
        x, y = d.x.copy(), d.y.copy()
        x[:k], y[:k] = rng.random(k) * room_x, rng.random(k) * room_y
        far = x.copy()
        far[:k] = np.minimum(x[:k] + 7.3 * d.die_w / m, room_x)
        for px, py in ((d.x, d.y), (x, y), (far, y)):   # the order stays the one of the start
            o.set_positions(px, py)
            g.set_positions(px, py)
            _, ovo = o.compute_potential(0)
            _, ovg = g.compute_potential(0)
            assert np.array_equal(g.array("DENSITY_I64"), o.get("density_i64"))
            assert abs(ovg - ovo) <= 1e-6 * max(abs(ovo), 1e-12)
    finally:
        g.close()
        o.close()
