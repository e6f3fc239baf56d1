"""Checkpoints and positions in device-mapped (pinned) host memory are read and
written by kernels, other memory by copies: the same state and the same bits
either way, on every alignment of the buffers and for every remainder of four
cells, with nothing written outside the arrays."""
import ctypes as C

import numpy as np
import pytest

from designs import small_synth

pytestmark = pytest.mark.gpu

F32P = C.POINTER(C.c_float)


def pinned(nbytes):
    import torch
    return torch.empty(nbytes, dtype=torch.uint8, pin_memory=True).numpy()


@pytest.mark.parametrize("cells", [900, 901, 902, 903, 5])
def test_mapped_and_other_memory_agree(cells):
    import reda_erplacer_gb300 as R
    p = R.Placement(small_synth(cells, seed=9, macros=2, io=30), (64, 64), 1.0, start_mode=1)
    p.run(3)
    blob = np.frombuffer(p.checkpoint(), np.uint8)
    start = [a.copy() for a in p.positions()]
    p.run(4)
    want = [a.copy() for a in p.positions()] + [p.array("PREV_X"), p.scalars()]
    for shift in (None, 0, 4, 8, 12, 1, 2):   # ordinary memory; pinned, on a boundary of floats or not
        if shift is None:
            at = blob.copy()
        else:
            at = pinned(blob.nbytes + 16)[shift:shift + blob.nbytes]
            at[:] = blob
        assert p.lib.erp_restore(p.h, at.ctypes.data, at.nbytes) == 0
        for a, b in zip(p.positions(), start):
            assert np.array_equal(a, b)
        p.run(4)
        for a, b in zip(p.positions(), want):
            assert np.array_equal(a, b)
        assert np.array_equal(p.array("PREV_X"), want[2]) and p.scalars() == want[3]
    n = p.N
    for ox, oy in ((0, 0), (1, 0), (0, 1), (1, 3)):
        x, y = (pinned(4 * (n + 8)).view(np.float32) for _ in range(2))
        x[:] = y[:] = -7.0
        u, v = x[ox:ox + n], y[oy:oy + n]
        assert p.lib.erp_get_positions(p.h, u.ctypes.data_as(F32P), v.ctypes.data_as(F32P)) == 0
        assert np.array_equal(u, want[0]) and np.array_equal(v, want[1])
        for buf, o in ((x, ox), (y, oy)):
            assert (buf[:o] == -7.0).all() and (buf[o + n:] == -7.0).all()
    p.close()


def test_registered_memory():
    """Arrays inside a registration of the caller's."""
    import torch
    import reda_erplacer_gb300 as R
    rt = torch.cuda.cudart()
    p = R.Placement(small_synth(5000, seed=3, macros=1, io=20), (64, 64), 1.0, start_mode=1)
    blob, n = np.frombuffer(p.checkpoint(), np.uint8), p.N
    p.run(2)
    want = [a.copy() for a in p.positions()]
    raw = np.zeros(blob.nbytes + 16384, np.uint8)
    raw = raw[(-raw.ctypes.data) % 4096:][:(blob.nbytes + 8192) // 4096 * 4096]
    assert int(rt.cudaHostRegister(raw.ctypes.data, raw.nbytes, 0)) == 0
    try:
        src = raw[-blob.nbytes:]   # ends with the registration
        src[:] = blob
        assert p.lib.erp_restore(p.h, src.ctypes.data, src.nbytes) == 0
        p.run(2)
        x, y = raw[:4 * n].view(np.float32), raw[-4 * n:].view(np.float32)
        assert p.lib.erp_get_positions(p.h, x.ctypes.data_as(F32P), y.ctypes.data_as(F32P)) == 0
        assert np.array_equal(x, want[0]) and np.array_equal(y, want[1])
    finally:
        assert int(rt.cudaHostUnregister(raw.ctypes.data)) == 0
    p.close()


@pytest.mark.parametrize("cells", [901, 900])
def test_positions_off_the_boundary_of_floats(cells):
    """Pinned arrays that start between two floats (a record's field, say) are copied:
    no kernel may store there.  Reading the positions, and a host-owned step."""
    import reda_erplacer_gb300 as R
    p = R.Placement(small_synth(cells, seed=9, macros=2, io=30), (64, 64), 1.0, start_mode=1)
    p.run(3)
    want = [a.copy() for a in p.positions()]
    n = p.N

    def at(shift):
        raw = pinned(4 * n + 16)
        raw[:] = 0xEE
        return raw, C.cast(raw.ctypes.data + shift, F32P), raw[shift:shift + 4 * n]

    for sx, sy in ((1, 0), (0, 2), (3, 1), (2, 2)):
        (rx, px, vx), (ry, py, vy) = at(sx), at(sy)
        assert p.lib.erp_get_positions(p.h, px, py) == 0
        assert vx.tobytes() == want[0].tobytes() and vy.tobytes() == want[1].tobytes()
        for raw, s in ((rx, sx), (ry, sy)):
            assert (raw[:s] == 0xEE).all() and (raw[s + 4 * n:] == 0xEE).all()
    blob = p.checkpoint()
    p.step()
    want = [a.copy() for a in p.positions()]
    p.restore(blob)
    assert p.lib.erp_get_positions(p.h, px, py) == 0
    assert p.lib.erp_step_host(p.h, px, py, None) == 0
    assert vx.tobytes() == want[0].tobytes() and vy.tobytes() == want[1].tobytes()
    p.close()


@pytest.mark.parametrize("shift", [0, 1, 4, 100])
def test_positions_into_arrays_that_share_memory(shift):
    """A caller that wants one coordinate may give one array for both, or two that
    overlap: y is written after x, in pinned memory as in any other."""
    import reda_erplacer_gb300 as R
    p = R.Placement(small_synth(20001, seed=9, macros=2, io=30), (64, 64), 1.0, start_mode=1)
    p.run(3)
    want, n = [a.copy() for a in p.positions()], p.N
    for buf in (np.zeros(n + shift, np.float32), pinned(4 * (n + shift)).view(np.float32)):
        for x, y in ((buf[:n], buf[shift:]), (buf[shift:], buf[:n])):
            assert p.lib.erp_get_positions(p.h, x.ctypes.data_as(F32P), y.ctypes.data_as(F32P)) == 0
            expect = np.concatenate([want[0][:shift], want[1]]) if y is not x and y.ctypes.data >= x.ctypes.data \
                else np.concatenate([want[1], want[0][n - shift:]])
            assert np.array_equal(buf, expect)
    p.close()
