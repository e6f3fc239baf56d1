"""The density scatter's three forms of a contribution's pieces (two of 21 bits, two of
23, three of 21), each on designs that take it by the bound of their contributions,
and on both sides of the item size from which 23 bits no longer leave room: the int64
map is the oracle's with all cells on one spot, within a few bins and spread out."""
import math

import numpy as np
import pytest

from designs import small_synth, spread_positions

pytestmark = pytest.mark.gpu


def form(d, m, n):
    """The form that the library's rule gives: the bound of a contribution in bits, and
    the cells of an item (a context run alone)."""
    k = d.num_movable
    w, h = d.w[:k].astype(np.float64), d.h[:k].astype(np.float64)
    shift = 61 - math.frexp(float(np.sum(w * h)))[1]
    bw, bh = d.die_w / m, d.die_h / n
    bits = math.log2((bw + (d.die_w + bw) * 2.0 ** -20) * (bh + (d.die_h + bh) * 2.0 ** -20)) + shift
    assert min(abs(bits - 42), abs(bits - 46)) > 0.01   # the bound's own small factors do not decide
    cap = max(-(-k // 608), 256)
    return "2x21" if bits < 42 else ("2x23" if bits < 46 and (cap + 31) // 32 * 32 <= 512 else "3x21")


@pytest.mark.parametrize("cells,m,n,want", [(1500, 64, 64, "3x21"), (40000, 128, 128, "3x21"), (700, 256, 512, "2x23"),
                                            (40000, 512, 512, "2x23"), (311000, 512, 512, "2x23"),
                                            (312000, 512, 512, "3x21"), (1500, 2048, 2048, "2x21"),
                                            (311500, 2048, 2048, "2x21")])
def test_every_form_gives_the_oracles_map(cells, m, n, want):
    import reda_erplacer_gb300 as R
    from oracle import erp_oracle as O
    d = small_synth(cells, seed=cells % 97, macros=1, io=8)
    assert form(d, m, n) == want
    o = O.Oracle(d, m, n, target_density=1.0, density_mode=O.DENSITY_FIXED, reduce_fp64=1)
    g = R.Placement(d, (m, n), 1.0)
    try:
        k = d.num_movable
        near = [c.copy() for c in (d.x, d.y)]
        rng = np.random.default_rng(cells)
        for c, size, die, bins in ((near[0], d.w, d.die_w, m), (near[1], d.h, d.die_h, n)):
            at = die / 2 - size[:k] / 2 + die / bins * rng.uniform(-5, 5, k)
            c[:k] = np.clip(at, 0, die - size[:k] - 1)
        one = [c.copy() for c in near]
        one[0][:k], one[1][:k] = np.float32(d.die_w / 2 + 0.3 * d.die_w / m), np.float32(d.die_h / 2 + 0.3 * d.die_h / n)
        for px, py in (one, near, spread_positions(d, seed=1, frac=0.95)):
            o.set_positions(px, py)
            g.set_positions(px, py)
            _, ovo = o.compute_potential(0)
            _, ovg = g.compute_potential(0)
            assert np.array_equal(g.array("DENSITY_I64"), o.get("density_i64"))
            assert abs(ovg - ovo) <= 1e-6 * max(abs(ovo), 1e-12)
    finally:
        g.close()
        o.close()
