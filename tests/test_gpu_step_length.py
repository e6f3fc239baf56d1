"""The step length that every block of the position update derives from the
gradient pass's block sums, at the edges of the blocks (four cells per thread, a
scalar tail, 1024 cells per block): a step against its stages, which sum in the
same groups, and the same bits in every block (the moves of all cells follow one
alpha and beta).

At iteration 0 the density weight of the two may differ by an ulp of FP32, 6e-8 of
a gradient; the step length divides by differences of gradients, of which 1e-2 or
more is left in two neighbouring steps from a spread start, so 1e-4 bounds it."""
import numpy as np
import pytest

from designs import small_synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [9, 10, 11, 1019, 1022, 1023, 1025, 2049, 5003])
def test_step_length(cells):
    import reda_erplacer_gb300 as R
    d = small_synth(cells, seed=cells, macros=1, io=20)
    a, b = (R.Placement(d, (64, 64), 1.0, start_mode=1) for _ in range(2))
    k = d.num_movable
    for it in range(3):
        x0, y0 = a.positions()
        px, py = a.array("PREV_X"), a.array("PREV_Y")
        a.step()
        hpwl = b.compute_hpwl(b.scalars()["gamma"])
        _, ovf = b.compute_potential(it, want_energy=False)
        b.step_adaptive(it)
        got, want = a.scalars(), b.scalars()
        b.scheduler_update(hpwl, ovf)
        assert got["alpha"] > 0 and abs(got["alpha"] - want["alpha"]) <= 1e-4 * want["alpha"]
        assert abs(got["beta"] - want["beta"]) <= 1e-6 * abs(want["beta"])
        assert got["alpha"] == np.float32(a.last_stats["alpha"])
        al, be = np.float32(got["alpha"]), np.float32(got["beta"])
        for now, old, prev, g, size, die in ((a.positions()[0], x0, px, a.array("PREV_GX"), d.w, d.die_w),
                                             (a.positions()[1], y0, py, a.array("PREV_GY"), d.h, d.die_h)):
            hi = np.float32(die) - size[:k] - np.float32(1)
            step = (old + be * (old - prev))[:k] - al * g[:k]
            assert np.array_equal(now[:k], np.where(step < 0, np.float32(0), np.where(step > hi, hi, step)))
    a.close()
    b.close()
