"""The Lorentz fields leave out the division of a zero by a positive number and
nothing else: J and B (kernels.py:1358-1383, 1438-1475) of potentials, conductivities
and bins that hold zeros of both signs, infinities and NaN equal the oracle's,
NaN for NaN, with four cells per thread and with one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(3, 5, 8), (7, 4, 36), (5, 6, 31), (2, 3, 1)]
ODD = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 1e-45, 3e38], np.float32)


def _plant(rng, a, every):
    flat = a.reshape(-1)
    for t in range(0, flat.size, every):
        flat[t] = ODD[rng.integers(ODD.size)]
    return a


@pytest.mark.parametrize("dx", [2e-4, 0.0, -2e-4])
@pytest.mark.parametrize("shape", SHAPES)
def test_current_density(shape, dx):
    import torch
    from oracle import oracle as O
    from waam_solver_b200 import kernels as K
    rng = np.random.default_rng(sum(shape))
    flags = rng.choice(np.array([0, 1, 2, 4], np.int32), size=shape).astype(np.int32)
    phi = _plant(rng, np.where(rng.random(shape) < 0.5, 0.0, rng.normal(size=shape)).astype(
        np.float32), 5)
    sigma = _plant(rng, rng.uniform(1e5, 1e6, shape).astype(np.float32), 11)
    want = [np.zeros(shape, np.float32) for _ in range(3)]
    O.call("wo_elec_compute_J", *want, phi, sigma, flags, *shape, dx)
    dev = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
    got = [torch.full(shape, 7.0, device="cuda") for _ in range(3)]
    K.elec_compute_J(*got, dev(phi), dev(sigma), dev(flags), dx, 2, *shape)
    for g, w in zip(got, want):
        assert np.array_equal(g.cpu().numpy(), w, equal_nan=True)


@pytest.mark.parametrize("dx", [2e-4, 0.0])
@pytest.mark.parametrize("arc", [(1.0, 2.0), (1.3, 2.2), (1.0 + 5e-4, 2.0)])
@pytest.mark.parametrize("shape", SHAPES)
def test_self_field(shape, arc, dx):
    import torch
    from oracle import oracle as O
    from waam_solver_b200 import kernels as K
    n_bins = 9
    rng = np.random.default_rng(sum(shape))
    bins = _plant(rng, np.where(rng.random((shape[2], n_bins)) < 0.4, 0.0, rng.normal(
        size=(shape[2], n_bins))).astype(np.float32), 4)
    want = [np.zeros(shape, np.float32) for _ in range(3)]
    O.call("wo_elec_B_axisymmetric", *want, bins, *shape, *arc, dx, 0.7, 1.2566e-6, n_bins)
    got = [torch.full(shape, 7.0, device="cuda") for _ in range(3)]
    K.elec_B_axisymmetric(*got, torch.from_numpy(bins).cuda(), *arc, dx, 0.7, 1.2566e-6, n_bins,
                          shape[2])
    for g, w in zip(got, want):
        assert np.array_equal(g.cpu().numpy(), w, equal_nan=True)
