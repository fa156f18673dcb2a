"""The Lorentz field kernels on grids of more than 2^27 columns or levels, where
one warp for each is more than 2^32 threads: the last columns against the same
columns of a small grid (the arc shifted by a whole number of cells, so that
every distance is the same float), the levels against their own sums."""
import pytest

pytestmark = pytest.mark.gpu

NX, NY = 16385, 8192            # 2^27 + 8192 columns of one cell
ROWS = 16                       # the x planes that are compared


def _grid(nx, fill):
    import torch
    return torch.full((nx, NY, 1), fill, dtype=torch.float32, device="cuda")


def test_self_field_of_the_last_columns():
    import torch
    from waam_solver_b200 import kernels as K
    bins = torch.rand((1, 64), device="cuda", generator=torch.Generator("cuda").manual_seed(3)) + 1.0
    out = []
    for nx in (NX, ROWS):
        B = [_grid(nx, float("nan")) for _ in range(3)]
        K.elec_B_axisymmetric(*B, bins, nx - 5.75, 4000.25, 2e-4, 90.0, 1.2566e-6, 64, 1)
        out.append([b[-ROWS:].clone() for b in B])
        assert not any(bool(torch.isnan(b).any()) for b in B)
    assert bool((out[0][0] != 0.0).any())
    for a, b in zip(*out):
        assert torch.equal(a, b)


def test_current_density_of_the_last_columns():
    import torch
    from waam_solver_b200 import kernels as K
    gen = torch.Generator("cuda").manual_seed(5)
    tail = torch.rand((ROWS + 1, NY, 1), device="cuda", generator=gen)
    out = []
    for nx in (NX, ROWS + 1):
        phi, sigma = _grid(nx, 0.0), _grid(nx, 1e6)
        phi[-ROWS - 1:] = tail
        flags = torch.zeros((nx, NY, 1), dtype=torch.int32, device="cuda")
        flags[-ROWS:, ::7] = 2
        J = [_grid(nx, float("nan")) for _ in range(3)]
        K.elec_compute_J(*J, phi, sigma, flags, 2e-4, 2, nx, NY, 1)
        out.append([j[-ROWS:].clone() for j in J])      # the plane before them is in both grids
        assert not any(bool(torch.isnan(j).any()) for j in J)
    for a, b in zip(*out):
        assert torch.equal(a, b)


def test_arc_source_of_the_last_columns():
    import torch
    from waam_solver_b200 import kernels as K
    out = []
    for nx in (NX, 4 * ROWS):
        src = _grid(nx, float("nan"))
        K.elec_arc_source(src, nx - 5.75, 4000.25, 0.5, 3.0, 140.0, 2e-4)
        assert not bool(torch.isnan(src).any())
        out.append(src[-ROWS:].clone())
    assert bool((out[0] > 0.0).any())
    # the scale divides by a double sum taken in another order: one unit of
    # float32 in the sum, one in the quotient
    assert bool(((out[0] - out[1]).abs() <= 2.0 ** -22 * out[1].abs()).all())


def test_arc_source_on_the_most_columns():
    """65534 x 32769 columns of one cell (2^31 - 2): the weight sum's stride past
    the last column does not fit 31 bits."""
    import torch
    from waam_solver_b200 import _native
    nx, ny = 65534, 32769
    out = []
    for m in (nx, 64):
        src = torch.empty((m, ny, 1), dtype=torch.float32, device="cuda")
        src[-ROWS:].fill_(float("nan"))
        ws = torch.zeros(int(_native.lib().waam_workspace_bytes(m * ny)), dtype=torch.uint8,
                         device="cuda")
        _native.call("waam_elec_arc_source", src.data_ptr(), m, ny, 1, m - 5.75, 4000.25, 0.5, 3.0,
                     140.0, 2e-4, ws.data_ptr(), ws.numel(), _native.stream_handle())
        out.append(src[-ROWS:].clone())
        del src, ws
        torch.cuda.empty_cache()
    assert bool((out[0] > 0.0).any())
    assert bool(((out[0] - out[1]).abs() <= 2.0 ** -22 * out[1].abs()).all())


def test_bin_prefix_of_the_last_levels():
    import torch
    from waam_solver_b200 import kernels as K
    nz = 2 ** 27 + 100
    bins = torch.rand((nz, 2), device="cuda", generator=torch.Generator("cuda").manual_seed(9))
    want = torch.stack((bins[:, 0], bins[:, 0] + bins[:, 1]), dim=1)
    K.elec_prefix_bins(bins, 2, nz)
    assert torch.equal(bins, want)
