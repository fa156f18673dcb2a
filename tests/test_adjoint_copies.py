"""The adjoint's state copies go by address only where that is what copy_ does:
a pair of another shape, type or memory order is converted by copy_, or refused
by it, and no row of the native table leaves its tensors (the entry point only
notes its rows here)."""
import ctypes
import types

import pytest
import torch

from waam_solver_b200 import _native, adjoint


class Rows(list):
    def copy_all(self):
        for dst, src, size in self:
            ctypes.memmove(dst, src, size)


@pytest.fixture
def rows(monkeypatch):
    sent = Rows()

    def call(name, table, count, stream):
        assert name == "waam_copy_planes"
        assert count <= _native.MAX_COPY_PLANES
        part = table._obj
        for q in range(count):
            sent.append((part[q].dst, part[q].src, part[q].bytes))

    monkeypatch.setattr(adjoint, "_call", call)
    monkeypatch.setattr(adjoint, "_stream", lambda: 0)
    monkeypatch.setattr(adjoint, "_device", lambda: -1, raising=False)     # the CPU's
    return sent


def test_plain_pairs_go_by_address(rows):
    src = [torch.rand(3, 5), torch.arange(7, dtype=torch.int32), torch.rand(())] * 13
    dst = [torch.zeros_like(t) for t in src]
    adjoint._copy_planes(list(zip(dst, src)))
    assert len(rows) == len(src)
    rows.copy_all()
    assert all(torch.equal(a, b) for a, b in zip(dst, src))


@pytest.mark.parametrize("shape", [(4, 4), (3,), (5, 3)])
def test_another_shape_raises_and_copies_nothing(rows, shape):
    whole, other = torch.zeros(2), torch.rand(shape)
    with pytest.raises(RuntimeError, match="size|shape"):
        adjoint._copy_planes([(whole, torch.ones(2)), (torch.zeros(3, 5), other)])
    assert rows == [] and not whole.any()


def test_other_types_and_orders_go_through_copy(rows):
    a, b, c = torch.zeros(2, 3), torch.zeros(3, 2), torch.zeros(5, dtype=torch.uint8)
    x = torch.rand(2, 3, dtype=torch.float64)
    y = torch.rand(2, 3).t()
    z = torch.arange(5, dtype=torch.uint8)          # five bytes: not a whole word
    adjoint._copy_planes([(a, x), (b, y), (c, z)])
    assert rows == []
    assert torch.equal(a, x.float()) and torch.equal(b, y) and torch.equal(c, z)


def test_copies_alike_are_checked_at_their_source(rows):
    src = [torch.rand(3, 5), torch.rand(4, 6).t(), torch.arange(5, dtype=torch.uint8)]
    dst = [torch.empty_like(t) for t in src]
    adjoint._copy_planes(zip(dst, src), alike=True)
    assert len(rows) == 1
    rows.copy_all()
    assert all(torch.equal(a, b) for a, b in zip(dst, src))


def _grid(n=24, **other):
    f = lambda: torch.rand(n)  # noqa: E731
    g = types.SimpleNamespace(n_cells=n, device=torch.device("cpu"), H=f(), T=f(), H_next=f(),
                              T_next=f(), f_l=f(), phi=f(), ux=f(), uy=f(), uz=f(),
                              flags=torch.zeros(n, dtype=torch.int32), step_scalars=torch.rand(16),
                              _cur=0)
    vars(g).update(other)
    return g


def test_tape_records_every_field(rows):
    g = _grid()
    tape = adjoint._Tape(g, 3, 24)
    tape.record(g, 1)
    rows.copy_all()
    for name, t in (("H", g.H), ("T", g.T), ("fl", g.f_l), ("phi", g.phi), ("flags", g.flags),
                    ("scal", g.step_scalars)):
        assert torch.equal(getattr(tape, name)[1], t), name
    assert torch.equal(tape.u[1], torch.stack((g.ux, g.uy, g.uz)))


@pytest.mark.parametrize("other", [dict(phi=torch.rand(25)), dict(flags=torch.rand(24)),
                                   dict(T=torch.rand(24, dtype=torch.float64)),
                                   dict(H_next=torch.rand(23)), dict(uy=torch.rand(48)[::2]),
                                   dict(step_scalars=torch.rand(17))])
def test_tape_refuses_fields_that_do_not_fit_its_slots(rows, other):
    with pytest.raises(_native.WaamError):
        adjoint._Tape(_grid(**other), 3, 24)
    assert rows == []


def test_tape_checks_the_fields_it_records(rows):
    g = _grid()
    tape = adjoint._Tape(g, 3, 24)
    g.f_l = torch.rand(30)          # the grid's field was replaced after the tape was made
    with pytest.raises(_native.WaamError):
        tape.record(g, 2)
    assert rows == []
