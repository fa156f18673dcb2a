"""The lagged stream of a pipelined step (kernels.py:2971-3010 on the cells that
the newer flags do not make active): bounced cells mended after the stores and
cells active in the next step left alone, on grids down to one cell and rows
beside a warp's 32, float32 and 2-byte elements, against the oracle's stream.

waam_step_finish runs it with an empty active list (no cell collides) and all
cells SOLID in the newest flags (the stream after it moves nothing)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (2, 1, 3), (1, 5, 33), (3, 9, 31), (4, 8, 32), (5, 7, 65), (3, 2, 97),
          (17, 1, 16)]
MIXES = [((0.4, 0.2, 0.3, 0.1), (0.3, 0.2, 0.4, 0.1)),    # FLUID, SOLID, GAS, IFACE: older, newer
         ((0.5, 0.5, 0.0, 0.0), (0.0, 0.0, 1.0, 0.0)),    # every streamed cell may bounce, none is left
         ((0.1, 0.3, 0.6, 0.0), (1.0, 0.0, 0.0, 0.0))]    # all are active next: nothing is written


@pytest.mark.parametrize("storage", [0, 1, 2])
@pytest.mark.parametrize("mix", MIXES)
@pytest.mark.parametrize("shape", SHAPES)
def test_lagged_stream_matches_the_oracle(shape, mix, storage):
    import torch
    from cases import OracleBackend
    from waam_solver_b200 import _native
    rng = np.random.default_rng(sum(shape) + 31 * MIXES.index(mix) + storage)
    n = int(np.prod(shape))
    kinds = np.array([0, 1, 2, 4], np.int32)
    older, newer = (rng.choice(kinds, size=shape, p=p).astype(np.int32) for p in mix)
    src, old = (rng.integers(0, 60000, (19,) + shape).astype(np.float32) for _ in range(2))
    to_dev = (lambda a: torch.from_numpy(a).cuda()) if storage == 0 else (
        lambda a: torch.from_numpy(a.astype(np.uint16).view(np.int16)).cuda())
    # after the buffer swap f_dst is what the lagged stream reads, f_src what it writes
    d_in, d_out = to_dev(src), to_dev(old)
    d_rr, d_r = torch.from_numpy(older).cuda(), torch.from_numpy(newer).cuda()
    solid = torch.ones(shape, dtype=torch.int32, device="cuda")
    dummy = torch.zeros((2, max(n, 16)), device="cuda")
    f = _native.WaamFields()
    for name, _ in _native.WaamFields._fields_[:24]:
        setattr(f, name, dummy[1 if name.endswith("_next") else 0].data_ptr())
    f.f_src, f.f_dst, f.flags = d_out.data_ptr(), d_in.data_ptr(), solid.data_ptr()
    f.flags_copy_rr, f.flags_copy_r = d_rr.data_ptr(), d_r.data_ptr()
    f.nx, f.ny, f.nz = shape
    p = _native.WaamStepParams()
    p.f_storage, p.stream_lag, p.collide_prev = storage, 1, 1
    ws = torch.zeros(int(_native.lib().waam_workspace_bytes(n)), dtype=torch.uint8, device="cuda")
    _native.call("waam_step_finish", ctypes.byref(f), ctypes.byref(p), ws.data_ptr(), ws.numel(),
                 _native.stream_handle())
    want = old.copy()
    OracleBackend().stream(src.copy(), want, older, *shape)
    left = np.isin(newer, (0, 4))
    want[:, left] = old[:, left]
    host = lambda t: t.cpu().numpy() if storage == 0 else (  # noqa: E731
        t.cpu().numpy().view(np.uint16).astype(np.float32))
    assert np.array_equal(host(d_out), want)
    assert np.array_equal(host(d_in), src)
