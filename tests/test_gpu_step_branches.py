"""The step graph's two branches (wirelength beside density and solve) against the
same stages called one after another, with every form of the solve and on both
sides of the size that decides which branch is captured first.

The totals are summed in other groupings (double-float, about 2^-44), and the
iteration-0 rescale likewise, so a scalar may differ by an ulp of FP32 and a
position by a few ulps of the die's size: the mean difference stays below 1e-6 of
it, 16 ulps.  A branch that ran ahead of its inputs is off by far more."""
import numpy as np
import pytest

from designs import small_synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells,precision", [(2000, 0), (2000, 1), (2000, 2), (60000, 2), (300000, 0), (300001, 0),
                                             (300001, 2)])
def test_step_equals_stages(cells, precision):
    import reda_erplacer_gb300 as R
    d = small_synth(cells, seed=9, macros=2, io=40)
    a = R.Placement(d, (128, 128), 1.0, start_mode=1, precision=precision)
    b = R.Placement(d, (128, 128), 1.0, start_mode=1, precision=precision)
    try:
        for it in range(3):
            a.step()
            hpwl = b.compute_hpwl(b.scalars()["gamma"])
            _, ovf = b.compute_potential(it, want_energy=False)
            b.step_adaptive(it)
            b.scheduler_update(hpwl, ovf)
            for got, want in ((a.last_stats["hpwl"], hpwl), (a.last_stats["overflow"], ovf)):
                assert abs(got - want) <= 1e-6 * abs(want)
        (xa, ya), (xb, yb) = a.positions(), b.positions()
        k = d.num_movable
        moved = np.abs(xb[:k] - d.x[:k]).mean() + np.abs(yb[:k] - d.y[:k]).mean()
        assert moved > 0
        scale = max(d.die_w, d.die_h)
        assert np.abs(xa - xb).mean() + np.abs(ya - yb).mean() <= 1e-6 * scale
    finally:
        a.close()
        b.close()
