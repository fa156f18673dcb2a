"""The reverse stream on the faces: y and z faces (up to three clamped
destinations beside the common one, the bounce-back from a clamped source) and
the periodic x wrap, on grids down to one cell.  Exact transpose of the forward
stream: <lam, S y> = <S^T lam, y>."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 3, 2), (3, 3, 1), (1, 4, 33), (5, 6, 32),
                                   (4, 9, 47)])
@pytest.mark.parametrize("p", [(0.3, 0.25, 0.35, 0.1), (0.8, 0.2, 0.0, 0.0), (0.1, 0.1, 0.8, 0.0)])
def test_reverse_stream_is_the_transpose(shape, p):
    import torch
    from waam_solver_b200 import _native
    n = int(np.prod(shape))
    rng = np.random.default_rng(n + int(100 * p[0]))
    flags = rng.choice([0, 1, 2, 4], size=n, p=p).astype(np.int32)
    # small integers: every float32 sum below is exact
    y = rng.integers(-8, 9, 19 * n).astype(np.float32)
    lam = rng.integers(-8, 9, 19 * n).astype(np.float32)
    seed = rng.integers(-8, 9, 19 * n).astype(np.float32)     # lam_yp on entry
    dev = lambda a: torch.from_numpy(a.copy()).cuda()  # noqa: E731
    fy, ff, fx = dev(y), dev(flags), torch.zeros(19 * n, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    _native.call("waam_stream", fy.data_ptr(), fx.data_ptr(), ff.data_ptr(), *shape, st)
    yp, xp, xn = dev(seed), dev(lam), torch.full((19 * n,), 7.0, device="cuda")
    _native.call("waam_adj_stream", yp.data_ptr(), xp.data_ptr(), xn.data_ptr(), ff.data_ptr(),
                 *shape, st)
    torch.cuda.synchronize()
    solid = np.tile(flags == 1, 19)
    lhs = float((lam * fx.cpu().numpy())[~solid].astype(np.float64).sum())
    rhs = float(((yp.cpu().numpy() - seed) * y).astype(np.float64).sum())
    assert lhs == rhs
    assert np.array_equal(xn.cpu().numpy(), np.where(solid, lam, np.float32(0.0)))


@pytest.mark.parametrize("count", [1, 31, 32, 33, 70])
def test_scatter_add_keeps_the_order_of_repeated_cells(count):
    import torch
    from waam_solver_b200 import _native
    rng = np.random.default_rng(count)
    cells = rng.integers(0, 12, count).astype(np.int32)
    vals = rng.normal(size=count).astype(np.float32)
    want = rng.normal(size=12).astype(np.float32)
    lam = torch.from_numpy(want.copy()).cuda()
    for c, v in zip(cells, vals):
        want[c] = np.float32(want[c] + v)
    dc, dv = torch.from_numpy(cells).cuda(), torch.from_numpy(vals).cuda()
    _native.call("waam_adj_scatter_add", lam.data_ptr(), dc.data_ptr(), dv.data_ptr(), count,
                 torch.cuda.current_stream().cuda_stream)
    assert np.array_equal(lam.cpu().numpy(), want)
