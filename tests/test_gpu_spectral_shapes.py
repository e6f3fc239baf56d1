"""The spectral solve's buffers: outputs on 4-byte boundaries only take scalar
stores, and asking for the potential adds blocks to the last pass.  Neither
changes a bit of the fields, and nothing is written outside the outputs.
(Accuracy: against the oracle in test_gpu_parity.py up to side 2048, here at 4096.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n", [(16, 16), (16, 64), (64, 16), (32, 4096), (64, 64), (64, 128), (128, 256), (256, 128),
                                 (256, 512), (512, 1024), (1024, 512), (2048, 64), (1024, 2048), (4096, 128),
                                 (128, 4096)])
def test_solve_buffers(m, n):
    import torch
    import reda_erplacer_gb300 as R
    rng = np.random.default_rng(m * 5 + n)
    rho = torch.from_numpy((0.7 + 0.3 * rng.random(m * n)).astype(np.float32))
    s = R.SpectralSolver(m, n, 1.3, 1.0, stream=torch.cuda.current_stream().cuda_stream)
    results = []
    for offset in (0, 1, 2):
        buf = [torch.zeros(m * n + 4, dtype=torch.float32, device="cuda") for _ in range(4)]
        at = [b[offset:offset + m * n] for b in buf]
        at[0].copy_(rho)
        for psi in (at[3].data_ptr(), None):
            s.solve(at[0].data_ptr(), at[1].data_ptr(), at[2].data_ptr(), psi)
            torch.cuda.synchronize()
            results.append([t.clone() for t in at[1:]])
        for b in buf[1:]:
            assert float(b[:offset].abs().sum()) == 0 and float(b[offset + m * n:].abs().sum()) == 0
    s.close()
    assert float(results[0][0].abs().sum()) > 0 and float(results[0][2].abs().sum()) > 0
    for r in results[1:]:
        for a, b in zip(results[0], r):
            assert torch.equal(a, b)


@pytest.mark.parametrize("m,n", [(64, 64), (64, 128), (128, 64), (128, 128)])
def test_small_grid_in_one_launch(m, n):
    """An isolated solve of a small grid is one launch of a cluster, a placement's is
    three launches: the same density gives the same bits, with and without the
    potential, twice in a row on the same intermediates."""
    import torch
    import reda_erplacer_gb300 as R
    from designs import small_synth
    p = R.Placement(small_synth(900, seed=m + 2 * n, macros=2), (m, n), 1.0, start_mode=1)
    p.compute_potential(0)
    rho, want = p.array("DENSITY"), [p.array(k) for k in ("FIELD_X", "FIELD_Y", "POTENTIAL")]
    info = p.scalars()
    p.close()
    src = torch.from_numpy(np.ascontiguousarray(rho)).cuda()
    s = R.SpectralSolver(m, n, info["bin_w"], info["bin_h"], stream=torch.cuda.current_stream().cuda_stream)
    for psi in (True, False, True):
        out = [torch.zeros(m * n, dtype=torch.float32, device="cuda") for _ in range(3)]
        s.solve(src.data_ptr(), out[0].data_ptr(), out[1].data_ptr(), out[2].data_ptr() if psi else None)
        torch.cuda.synchronize()
        for got, ref in list(zip(out, want))[:3 if psi else 2]:
            assert np.array_equal(got.cpu().numpy(), ref.reshape(-1))
    s.close()


@pytest.mark.parametrize("precision", [1, 2])
@pytest.mark.parametrize("m,n", [(128, 128), (128, 2048), (2048, 128), (256, 512), (1024, 1024), (2048, 2048)])
def test_contraction_tiles(m, n, precision):
    """The tensor-core solve at sizes that take every tile width, one tile per SM
    and several: the two fields are the same bits with and without the potential
    (other widths and other tiles per SM), on 32-byte and on 16-byte boundaries
    (other stores), and twice in a row (the ring and both accumulators in use
    again).  (Accuracy is tested in test_gpu_parity.py.)"""
    import torch
    import reda_erplacer_gb300 as R
    rng = np.random.default_rng(m + n)
    rho = torch.from_numpy((0.7 + 0.3 * rng.random(m * n)).astype(np.float32)).cuda()
    stream = torch.cuda.current_stream().cuda_stream
    s = R.SpectralSolver(m, n, 1.3, 1.0, stream=stream, precision=precision)
    results = []
    for offset in (0, 4, 0):
        buf = [torch.zeros(m * n + 8, dtype=torch.float32, device="cuda") for _ in range(3)]
        at = [b[offset:offset + m * n] for b in buf]
        for psi in (at[2].data_ptr(), None):
            s.solve(rho.data_ptr(), at[0].data_ptr(), at[1].data_ptr(), psi)
            torch.cuda.synchronize()
            results.append([t.clone() for t in at])
        for b in buf:
            assert float(b[:offset].abs().sum()) == 0 and float(b[offset + m * n:].abs().sum()) == 0
    s.close()
    for r in results[1:]:
        for a, b in zip(results[0], r):
            assert torch.equal(a, b)


@pytest.mark.parametrize("precision", [1, 2])
@pytest.mark.parametrize("m,n", [(128, 128), (256, 512), (1024, 2048)])
def test_contraction_outputs_on_4_byte_boundaries(m, n, precision):
    """The tensor-core solve into buffers that start on any boundary of floats, each
    its own: the bits of aligned ones, nothing written outside, the density where it
    is (BF16x3 takes it on 4-byte boundaries too)."""
    import torch
    import reda_erplacer_gb300 as R
    rng = np.random.default_rng(m + 3 * n)
    rho = torch.from_numpy((0.7 + 0.3 * rng.random(m * n)).astype(np.float32))
    s = R.SpectralSolver(m, n, 1.3, 1.0, stream=torch.cuda.current_stream().cuda_stream, precision=precision)
    want = None
    for offsets in ((0, 0, 0), (1, 0, 0), (0, 2, 3), (3, 1, 2), (2, 2, 2)):
        buf = [torch.full((m * n + 8,), -7.0, dtype=torch.float32, device="cuda") for _ in range(3)]
        at = [b[o:o + m * n] for b, o in zip(buf, offsets)]
        src = torch.zeros(m * n + 8, dtype=torch.float32, device="cuda")
        skip = offsets[0] if precision == 2 else 0
        src[skip:skip + m * n] = rho.cuda()
        s.solve(src[skip:].data_ptr(), *[t.data_ptr() for t in at])
        torch.cuda.synchronize()
        got = [t.clone() for t in at]
        want = want or got
        for a, b in zip(want, got):
            assert torch.equal(a, b)
        for b, o in zip(buf, offsets):
            assert bool((b[:o] == -7.0).all()) and bool((b[o + m * n:] == -7.0).all())
    s.close()


@pytest.mark.parametrize("precision,m,n", [(0, 64, 64), (0, 64, 128), (0, 128, 64), (0, 128, 128), (0, 16, 64),
                                           (0, 512, 256), (0, 4096, 64), (1, 256, 128), (2, 256, 128)])
def test_output_in_the_densitys_place(precision, m, n):
    """An output that overwrites the density (the density is read before any output is
    written, in one launch or several): the bits of outputs of their own."""
    import torch
    import reda_erplacer_gb300 as R
    rng = np.random.default_rng(m * 7 + n)
    rho = torch.from_numpy((0.7 + 0.3 * rng.random(m * n)).astype(np.float32)).cuda()
    s = R.SpectralSolver(m, n, 1.3, 1.0, stream=torch.cuda.current_stream().cuda_stream, precision=precision)
    want = [torch.empty_like(rho) for _ in range(3)]
    s.solve(rho.data_ptr(), *[t.data_ptr() for t in want])
    for which in range(3):
        out = [torch.empty_like(rho) for _ in range(3)]
        out[which].copy_(rho)
        s.solve(out[which].data_ptr(), *[t.data_ptr() for t in out])
        torch.cuda.synchronize()
        for a, b in zip(want, out):
            assert torch.equal(a, b)
    s.close()


@pytest.mark.parametrize("m,n", [(4096, 64), (64, 4096), (4096, 16), (4096, 2048), (2048, 4096)])
def test_side_4096_against_64_bits(m, n):
    """The longest transforms against the solve in 64 bits.  The bar is twice the error
    that the oracle's own FP32 solve has on the same density: both round every product
    and sum of transforms of the same lengths once, in other orders.  (An absolute bar
    does not serve: of a density of white noise around 0.85 the rounding of the mean is
    most of the error, and it grows with the grid.)"""
    import torch
    import reda_erplacer_gb300 as R
    from oracle import erp_oracle as O
    rng = np.random.default_rng(m * 3 + n)
    rho = torch.from_numpy((0.7 + 0.3 * rng.random((m, n))).astype(np.float32))
    want = O.poisson(rho.numpy().astype(np.float64), 1.3, 1.1, dtype=np.float64)
    fp32 = O.poisson(rho.numpy(), 1.3, 1.1, dtype=np.float32)
    s = R.SpectralSolver(m, n, 1.3, 1.1, stream=torch.cuda.current_stream().cuda_stream)
    src, out = rho.cuda(), [torch.empty(m, n, dtype=torch.float32, device="cuda") for _ in range(3)]
    s.solve(src.data_ptr(), *[t.data_ptr() for t in out])
    torch.cuda.synchronize()
    s.close()
    flat = [[np.asarray(t, np.float64).ravel() for t in three] for three in ([t.cpu().numpy() for t in out], fp32, want)]
    for got, theirs, ref in zip(*flat):
        assert np.linalg.norm(got - ref) <= 2 * np.linalg.norm(theirs - ref)
