"""The streaming and collision operators where their warps and blocks end.

* stream (kernels.py:2971-3010): rows shorter than, equal to and just over a
  warp's 32 cells, single planes and random flags of all four kinds, so that
  every solid-source vote (row, below, above, clamped and wrapped faces)
  decides; bit-exact against the oracle.
* collide_srt (kernels.py:2778-2885): the lattice sums without their zero
  products, on block remainders and with cells whose populations, forces or
  liquid fraction hold infinities and NaN; equal to the oracle, NaN for NaN.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def backends():
    from cases import OracleBackend
    from cuda_backend import CudaBackend
    return CudaBackend(), OracleBackend()


def _flags(rng, shape, p):
    return rng.choice(np.array([0, 1, 2, 4], np.int32), size=shape, p=p).astype(np.int32)


@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 1, 3), (1, 5, 33), (3, 9, 31), (4, 8, 32),
                                   (2, 17, 64), (5, 7, 65), (3, 2, 97)])
@pytest.mark.parametrize("p", [(0.4, 0.2, 0.3, 0.1), (0.9, 0.1, 0.0, 0.0), (0.0, 0.1, 0.9, 0.0)])
def test_stream_at_row_ends(backends, shape, p):
    cuda, oracle = backends
    rng = np.random.default_rng(sum(shape) * 7 + int(10 * p[0]))
    flags = _flags(rng, shape, p)
    src = rng.normal(size=(19,) + shape).astype(np.float32)
    got = rng.normal(size=(19,) + shape).astype(np.float32)
    want = got.copy()
    cuda.stream(src.copy(), got, flags, *shape)
    oracle.stream(src.copy(), want, flags, *shape)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("n", [1, 127, 128, 129, 1000])
@pytest.mark.parametrize("odd", [False, True])
def test_collide_srt_sums(backends, n, odd):
    cuda, oracle = backends
    rng = np.random.default_rng(n)
    shape = (1, 1, n)
    f = (1.0 / 19.0 + 0.01 * rng.normal(size=(19,) + shape)).astype(np.float32)
    F = (1e-3 * rng.normal(size=(3,) + shape)).astype(np.float32)
    fl = rng.uniform(0.0, 1.0, shape).astype(np.float32)
    flags = _flags(rng, shape, (0.6, 0.1, 0.1, 0.2))
    if odd:
        bad = np.array([np.nan, np.inf, -np.inf], np.float32)
        for t in range(0, n, 7):
            f[rng.integers(19), 0, 0, t] = bad[t % 3]
        F[rng.integers(3), 0, 0, 3::11] = np.inf
        fl[0, 0, 5::13] = np.nan
        f[:, 0, 0, 1::17] = 0.0
    out = []
    for b in (cuda, oracle):
        dst = np.zeros_like(f)
        mom = [np.zeros(shape, np.float32) for _ in range(4)]
        b.collide_srt(f.copy(), dst, *mom, F[0].copy(), F[1].copy(), F[2].copy(), fl.copy(), flags,
                      n, 1.7, 1.6e5)
        out.append([dst] + mom)
    for a, b in zip(*out):
        assert np.array_equal(a, b, equal_nan=True)


@pytest.mark.parametrize("storage", [0, 1])
@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 1, 3), (3, 9, 31), (4, 8, 32), (5, 7, 65),
                                   (3, 2, 97)])
def test_step_stream_at_row_ends(backends, storage, shape):
    """The fused step's stream in order, float32 and 2-byte elements, against the
    oracle's on the same values (beside the next step's stages it mends the
    bounced cells after its stores: test_gpu_lagged_stream.py)."""
    import ctypes
    import torch
    from waam_solver_b200 import _native
    _, oracle = backends
    rng = np.random.default_rng(sum(shape) + storage)
    n = int(np.prod(shape))
    flags = _flags(rng, shape, (0.4, 0.2, 0.3, 0.1))
    src, want = (rng.integers(0, 60000, (19,) + shape).astype(np.float32) for _ in range(2))
    to_dev = (lambda a: torch.from_numpy(a).cuda()) if storage == 0 else (
        lambda a: torch.from_numpy(a.astype(np.uint16).view(np.int16)).cuda())
    d_src, d_dst, d_flags = to_dev(src), to_dev(want), torch.from_numpy(flags).cuda()
    dummy = torch.zeros((2, max(n, 16)), device="cuda")
    f = _native.WaamFields()
    for name, kind in _native.WaamFields._fields_[:24]:
        setattr(f, name, dummy[1 if name.endswith("_next") else 0].data_ptr())
    f.f_src, f.f_dst, f.flags = d_src.data_ptr(), d_dst.data_ptr(), d_flags.data_ptr()
    f.nx, f.ny, f.nz = shape
    p = _native.WaamStepParams()
    p.f_storage = storage
    _native.call("waam_step_stream", ctypes.byref(f), ctypes.byref(p),
                 torch.cuda.current_stream().cuda_stream)
    oracle.stream(src, want, flags, *shape)
    got = d_dst.cpu().numpy()
    got = got if storage == 0 else got.view(np.uint16).astype(np.float32)
    assert np.array_equal(got, want)
