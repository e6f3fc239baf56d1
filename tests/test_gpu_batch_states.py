"""A batch arms, reads and disarms its instances' states in one launch each, and
captures the scatter-order refresh only when one is due: runs cut into pieces on
either side of the refresh interval give the bits of one long run and of the same
designs alone, an instance's queued work is seen, a run of no steps changes
nothing, and afterwards every instance steps on unarmed."""
import numpy as np
import pytest

from designs import small_synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 3, 5])
def test_batch_runs_in_pieces(count):
    import reda_erplacer_gb300 as R
    bins = [(64, 64), (32, 64), (128, 64), (64, 64), (128, 128)][:count]
    designs = [small_synth(700 + 300 * i, seed=60 + i, macros=1) for i in range(count)]
    pieces = (0, 1, 7, 40, 0, 33)
    b, whole = R.Batch(designs, bins, 1.0, start_mode=1), R.Batch(designs, bins, 1.0, start_mode=1)
    for k in pieces:
        done, last = b.run(k)
        assert list(done) == [k] * count
    whole.run(sum(pieces))
    for i, (d, mn) in enumerate(zip(designs, bins)):
        p = R.Placement(d, mn, 1.0, start_mode=1)
        p.run(sum(pieces))
        for u, v, w in zip(b.positions(i), whole.positions(i), p.positions()):
            assert np.array_equal(u, v) and np.array_equal(u, w)
        p.close()
        for _ in range(2):   # queued on the instance's own stream, not waited for
            assert b.lib.erp_step(b.lib.erp_batch_context(b.h, i), None) == 0
    whole.run(3)
    b.run(1)
    for i in range(count):
        for u, v in zip(b.positions(i), whole.positions(i)):
            assert np.array_equal(u, v)
    b.close()
    whole.close()
