"""waam_copy_planes: every listed array whole, nothing around it touched, on
sizes at and beside a block's share, aligned to 16 bytes and not."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(sizes, offs):
    import torch
    from waam_solver_b200 import _native
    rng = np.random.default_rng(len(sizes))
    rows = (_native.WaamCopyPlane * len(sizes))()
    kept = []
    for row, n, (so, do) in zip(rows, sizes, offs):
        src = rng.integers(-2**31, 2**31 - 1, n + 16, dtype=np.int64).astype(np.int32)
        s = torch.from_numpy(src).cuda()
        d = torch.full((n + 16,), 77, dtype=torch.int32, device="cuda")
        row.src, row.dst, row.bytes = s.data_ptr() + 4 * so, d.data_ptr() + 4 * do, 4 * n
        kept.append((src, s, d))
    _native.call("waam_copy_planes", ctypes.byref(rows), len(sizes),
                 torch.cuda.current_stream().cuda_stream)
    for (src, _, d), n, (so, do) in zip(kept, sizes, offs):
        want = np.full(n + 16, 77, np.int32)
        want[do:do + n] = src[so:so + n]
        assert np.array_equal(d.cpu().numpy(), want)


@pytest.mark.parametrize("offs", [(0, 0), (4, 8), (1, 0), (0, 3), (1, 1)])
def test_sizes_and_alignments(offs):
    sizes = [1, 3, 4, 5, 0, 4095, 4096, 4097, 8192, 12291]
    _run(sizes, [offs] * len(sizes))


@pytest.mark.parametrize("count", [1, 32])
def test_table_sizes(count):
    _run([17 + 4096 * (q % 3) for q in range(count)], [(0, 0)] * count)


def test_bad_tables_are_refused():
    import torch
    from waam_solver_b200 import _native
    t = torch.zeros(16, device="cuda")
    ok = dict(dst=t.data_ptr(), src=t.data_ptr() + 32, bytes=16)
    st = torch.cuda.current_stream().cuda_stream
    for bad in (dict(bytes=6), dict(bytes=-4), dict(dst=None), dict(src=None),
                dict(dst=t.data_ptr() + 2)):
        row = _native.WaamCopyPlane(**dict(ok, **bad))
        with pytest.raises(_native.WaamError):
            _native.call("waam_copy_planes", ctypes.byref(row), 1, st)
    many = (_native.WaamCopyPlane * 33)()
    with pytest.raises(_native.WaamError):
        _native.call("waam_copy_planes", ctypes.byref(many), 33, st)
