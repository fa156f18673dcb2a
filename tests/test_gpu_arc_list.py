"""The fused step's arc weight sum and injection over the tile list, on lists at
and beside what their blocks, their share of tiles and their batches take, with
partial tiles and beyond the shared tables (nz > 1024, nx + ny + nz > 3072),
against the oracle's injection (kernels.py:443-510, 548-622).

The sum is a double sum in another order, rounded to float32: one unit in the
last place of it, one more in the energy per weight and in each product."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ULP = 2.0 ** -23
# (nx, ny, nz): tiles of 32 k by 8 j, all of them listed (148, 1184 and 4736
# tiles, where the grid's size turns, and two beside them; the last two beyond
# the depth table and the axis tables)
SHAPES = [(1, 1, 33), (1, 8, 33), (4, 5, 40), (73, 8, 64), (74, 3, 50), (75, 8, 64), (591, 8, 40),
          (592, 8, 36), (593, 6, 33), (2367, 8, 33), (2368, 8, 40), (2369, 3, 40), (60, 60, 45),
          (3, 17, 1030), (3100, 8, 40)]
ARC = dict(Q_w=3000.0, eta=0.75, dt=1e-5, dx3=8e-12, pen=4.0)
AXES = dict(sign=1.0, ff=0.6, fr=1.4, a_f=9.0, a_r=21.0, gb=4.0, gc=3.0)


def _run(shape, flags, f_l, phi, kind, pos):
    import torch
    from waam_solver_b200 import _native
    n = int(np.prod(shape))
    nx, ny, nz = shape
    kt, jt = (nz + 31) // 32, (ny + 7) // 8
    tiles = kt * jt * nx
    dev = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
    dummy = torch.zeros((2, max(n, 16)), device="cuda")
    f = _native.WaamFields()
    for name, _ in _native.WaamFields._fields_[:24]:
        setattr(f, name, dummy[1 if name in ("f_dst", "H_next", "T_next") else 0].data_ptr())
    H, scal = torch.zeros(n, device="cuda"), torch.zeros(16, device="cuda")
    scal[4], scal[5] = pos
    keep = [dev(flags), dev(f_l), dev(phi), H, scal,
            torch.zeros(kt * nx * ny + tiles, dtype=torch.uint8, device="cuda"),
            torch.zeros(1 + tiles, dtype=torch.int32, device="cuda"),
            torch.full((tiles,), float("nan"), dtype=torch.float64, device="cuda"),
            torch.zeros(int(_native.lib().waam_workspace_bytes(n)), dtype=torch.uint8,
                        device="cuda")]
    f.flags, f.f_l, f.phi, f.H, f.step_scalars, f.tile_bits, f.tile_list, f.tile_part = (
        t.data_ptr() for t in keep[:8])
    f.nx, f.ny, f.nz = shape
    p = _native.WaamStepParams()
    p.welding, p.arc_kind, p.surface_weighting, p.nz_solid = 1, kind, 1, 8
    p.sigma_heat, p.arc_k_offset = 5.0, 0.0
    for k, v in dict(ARC, **AXES).items():
        setattr(p, k, v)
    _native.call("waam_step_pre", ctypes.byref(f), ctypes.byref(p), keep[8].data_ptr(),
                 keep[8].numel(), _native.stream_handle())
    assert int(keep[6][0].item()) == tiles
    return scal.cpu().numpy(), H.cpu().numpy().reshape(shape)


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("shape", SHAPES)
def test_list_sum_and_injection_match_the_oracle(shape, kind):
    from oracle import oracle as O
    rng = np.random.default_rng(sum(shape) + kind)
    nx, ny, nz = shape
    flags = rng.choice(np.array([0, 1, 2, 4], np.int32), size=shape, p=[0.3, 0.3, 0.3, 0.1])
    flags[:, :, nz // 2:] = 2
    flags[:, :, 0] = 1
    f_l = rng.uniform(0.0, 1.0, shape).astype(np.float32)
    phi = np.where(flags == 2, 0.0, 1.0).astype(np.float32)
    pos = (0.6 * nx, 0.4 * ny)
    flags = flags.astype(np.int32)
    scal, H = _run(shape, flags, f_l, phi, kind, pos)
    again = _run(shape, flags, f_l, phi, kind, pos)
    assert np.array_equal(scal, again[0]) and np.array_equal(H, again[1])
    want = np.zeros(shape, np.float32)
    arc = (float(scal[4]), float(scal[5]), float(scal[0]))
    a = ARC
    if kind == 0:
        total = O.call("wo_inject_arc_heat", want, flags, f_l, nx, ny, nz, *arc, a["Q_w"], 5.0,
                       a["dt"], a["dx3"], a["eta"], a["pen"], 1)
    else:
        total = O.call("wo_inject_goldak_heat", want, flags, f_l, nx, ny, nz, *arc, a["Q_w"],
                       a["dt"], a["dx3"], a["eta"], *(AXES[k] for k in (
                           "sign", "ff", "fr", "a_f", "a_r", "gb", "gc")), a["pen"], 1)
    assert total > 0.0
    assert abs(float(scal[1]) - total) <= ULP * total
    assert np.all(np.abs(H - want) <= 4.0 * ULP * np.abs(want) + 2.0 ** -126)   # (subnormal: by its step)
