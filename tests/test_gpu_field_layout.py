"""The two field layouts between the solve and the force: interleaved for large
designs and packed batches, two maps otherwise.  A batch's packed instances
(interleaved) give the bits of the same designs run alone (two maps), on every
transform of the packed sides, with cells wider than two bins among them; a
design on either side of the size rule has its fields and force at the oracle's."""
import numpy as np
import pytest

from designs import small_synth

pytestmark = pytest.mark.gpu


def widened(d, every, width):
    d.w[:d.num_movable:every] = width
    d.x[:d.num_movable] = np.clip(d.x[:d.num_movable], 0, d.die_w - d.w[:d.num_movable] - 1)
    d.movable_area = float(np.sum(d.w[:d.num_movable].astype(np.float64) * d.h[:d.num_movable]))
    return d


def test_packed_batch_equals_alone():
    import reda_erplacer_gb300 as R
    bins = [(64, 64), (128, 64), (64, 256), (256, 128), (256, 256)]
    designs = [widened(small_synth(900 + 700 * i, seed=40 + i, macros=i), 53, 6.0) for i in range(5)]
    b = R.Batch(designs, bins, 1.0, start_mode=1)
    assert b.packed_instances() == 5
    b.run(20)
    for i, (d, mn) in enumerate(zip(designs, bins)):
        p = R.Placement(d, mn, 1.0, start_mode=1)
        p.run(20)
        for a, c in zip(p.positions(), b.positions(i)):
            assert np.array_equal(a, c)
        p.close()
    b.close()


@pytest.mark.parametrize("cells", [131071, 131072])
def test_fields_and_force_at_the_size_rule(cells):
    import reda_erplacer_gb300 as R
    from oracle import erp_oracle as O
    d = widened(small_synth(cells, seed=5, macros=2, io=40), 211, 9.0)
    o = O.Oracle(d, 256, 256, target_density=1.0, start_mode=O.START_DB, density_mode=O.DENSITY_FIXED, reduce_fp64=1)
    g = R.Placement(d, (256, 256), 1.0, start_mode=1)
    try:
        o.compute_potential(0)
        g.compute_potential(0)
        for mine, theirs in (("FIELD_X", "field_x"), ("FIELD_Y", "field_y"), ("POTENTIAL", "potential"),
                             ("DENS_GRAD_X", "dens_grad_x"), ("DENS_GRAD_Y", "dens_grad_y")):
            a, r = g.array(mine).astype(np.float64), o.get(theirs).astype(np.float64)
            assert np.linalg.norm(a - r) <= 1e-5 * np.linalg.norm(r), mine   # the parity bar of fields and force
    finally:
        g.close()
        o.close()


def test_interleaved_fields_read_back():
    """The fields of an interleaved context, as maps: the bits of the same design's two
    maps, into ordinary and page-locked arrays, x and y in either order; a short
    destination is refused; the solve's scratch that the maps pass through is free for
    the next step."""
    import ctypes as C
    import torch
    import reda_erplacer_gb300 as R
    bins = [(64, 64), (64, 128), (256, 64), (128, 128)]
    designs = [small_synth(800 + 300 * i, seed=70 + i, macros=1) for i in range(4)]
    b = R.Batch(designs, bins, 1.0, start_mode=1)
    assert b.packed_instances() == 4
    for steps in (5, 4):
        b.run(steps)
    for i, (d, (m, n)) in enumerate(zip(designs, bins)):
        p = R.Placement(d, (m, n), 1.0, start_mode=1)
        p.run(9)
        ctx = C.c_void_p(b.lib.erp_batch_context(b.h, i))
        pinned = torch.empty(m * n, pin_memory=True).numpy()
        for name in ("FIELD_Y", "FIELD_X", "FIELD_Y"):
            want = p.array(name)
            for out in (np.zeros(m * n, np.float32), pinned):
                out[:] = -7.0
                to = out.ctypes.data_as(C.c_void_p)
                assert b.lib.erp_get_array(ctx, R.lib.ARR[name], to, out.nbytes - 4) == R.lib.EINVAL
                assert (out == -7.0).all()
                assert b.lib.erp_get_array(ctx, R.lib.ARR[name], to, out.nbytes) == 0
                assert np.abs(want).max() > 0 and np.array_equal(out, want)
            b.lib.erp_step(ctx, None)
            p.step()
        for u, v in zip(b.positions(i), p.positions()):
            assert np.array_equal(u, v)
        p.close()
    b.close()
