"""The Lorentz fields' kernels take four cells per thread where nz is a multiple
of four and every field starts on 16 bytes, else one: both forms on the same
grids (fields moved off their 16 bytes force the second), bit for bit, and the
live and newly fixed lists against the mask."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _shifted(shape, off, dtype, fill=None):
    """A contiguous tensor of `shape` whose storage starts `off` elements in."""
    import torch
    n = int(np.prod(shape))
    t = torch.zeros(n + 16, dtype=dtype, device="cuda")[off:off + n].view(shape)
    if fill is not None:
        t.copy_(torch.from_numpy(fill))
    return t


def _state(shape, seed):
    rng = np.random.default_rng(seed)
    flags = rng.choice(np.array([0, 1, 2, 4], np.int32), size=shape, p=[0.2, 0.2, 0.5, 0.1])
    flags[:, :, shape[2] // 2:] = 2
    f_l = rng.uniform(0.0, 1.0, shape).astype(np.float32)
    phi = rng.normal(size=shape).astype(np.float32)
    fixed = (rng.random(shape) < 0.5).astype(np.uint8)
    return flags.astype(np.int32), f_l, phi, fixed


def _fields(shape, seed, off):
    import torch
    from waam_solver_b200 import _native, kernels as K
    flags, f_l, phi, fixed = _state(shape, seed)
    f32 = torch.float32
    n = int(np.prod(shape))
    mk = lambda fill=None: _shifted(shape, off, f32, fill)  # noqa: E731
    d_flags, d_fl, d_phi = _shifted(shape, off, torch.int32, flags), mk(f_l), mk(phi)
    d_fixed = _shifted(shape, 3 * off, torch.uint8, fixed)
    sigma, phi_b = mk(), mk(phi)
    live, zero = (torch.zeros(n, dtype=torch.int32, device="cuda") for _ in range(2))
    counts = torch.zeros(int(_native.lib().waam_elec_counts_len(*shape)), dtype=torch.int32,
                         device="cuda")
    K.elec_prepare(sigma, d_fixed, phi_b, d_fl, d_flags, 1e6, 1e5, 3, live, zero, counts)
    J = [mk() for _ in range(3)]
    K.elec_compute_J(*J, d_phi, sigma, d_flags, 2e-4, 2, *shape)
    B = [mk() for _ in range(3)]
    bins = torch.from_numpy(np.random.default_rng(1).normal(size=(shape[2], 40)).astype(np.float32)).cuda()
    K.elec_prefix_bins(bins, 40, shape[2])
    K.elec_B_axisymmetric(*B, bins, 3.3, 2.2, 2e-4, 0.5, 1.2566e-6, 40, shape[2])
    src = mk()
    K.elec_arc_source(src, 3.3, 2.2, 5.0, 4.5, 140.0, 2e-4)
    c = counts.cpu().numpy()
    out = [t.cpu().numpy().copy() for t in (sigma, d_fixed, phi_b, *J, *B, src, bins)]
    lists = live.cpu().numpy()[:c[0]], np.sort(zero.cpu().numpy()[:c[1]])
    # the lists are the mask's
    k = np.arange(shape[2])
    new = ((flags == 2) | ((flags == 1) & (k <= 3))).reshape(-1)
    assert np.array_equal(out[1].reshape(-1) != 0, new)
    assert np.array_equal(lists[0], np.nonzero(~new)[0])
    assert np.array_equal(lists[1], np.nonzero(new & (fixed.reshape(-1) == 0))[0])
    return out


@pytest.mark.parametrize("shape", [(1, 1, 4), (3, 5, 8), (7, 9, 32), (5, 6, 36), (8, 8, 64),
                                   (3, 7, 31), (2, 3, 1)])
def test_both_forms_agree(shape):
    a, b = _fields(shape, 5, 0), _fields(shape, 5, 1)
    for x, y in zip(a, b):
        assert np.array_equal(x, y)
