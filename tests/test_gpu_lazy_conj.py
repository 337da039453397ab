"""GPU: inputs and cotangents that torch holds as lazy conjugate or negative views
(`c.conj()`, `z.conj().imag`) are read as the values they stand for: every result
equals that of the same values stored plainly (the same kernels on the same numbers,
so within the atomics' float order, 1e-6 for complex64)."""

import pytest
import torch

import nufftax_b200 as nb
from nufftax_b200._plan import PointSort
from nufftax_b200.batch import BatchPlan

pytestmark = pytest.mark.gpu

N, M = (24, 20), 700


def _data():
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    z = torch.rand((2, M), generator=g, device="cuda") * 6 - 3
    c = torch.randn(M, generator=g, device="cuda", dtype=torch.complex64)
    f = torch.randn(N[::-1], generator=g, device="cuda", dtype=torch.complex64)
    t = torch.rand((2, 300), generator=g, device="cuda") * 20 - 10
    return list(z), c, f, list(t)


def _neg(x):
    """x as a lazily negated view."""
    v = torch.complex(torch.zeros_like(x), -x).conj().imag
    assert v.is_neg()
    return v


def _close(a, b):
    assert torch.linalg.norm(a - b) <= 1e-6 * torch.linalg.norm(b)


def test_strengths_modes_and_coordinates():
    x, c, f, t = _data()
    lc, lf = c.conj().resolve_conj().conj(), f.conj().resolve_conj().conj()
    assert lc.is_conj() and lf.is_conj()
    xn, tn = [_neg(v) for v in x], [_neg(v) for v in t]
    _close(nb.nufft2d1(*x, lc, N), nb.nufft2d1(*x, c, N))
    _close(nb.nufft2d1(*xn, c, N), nb.nufft2d1(*x, c, N))
    _close(nb.nufft2d2(*x, lf), nb.nufft2d2(*x, f))
    g = nb.compute_type3_grid_sizes_2d(3.0, 3.0, 10.0, 10.0)
    _close(nb.nufft2d3(*xn, lc, *tn, g), nb.nufft2d3(*x, c, *t, g))


def test_cotangents():
    x, c, f, _ = _data()
    for wrap in (lambda v: v.conj(), lambda v: v.conj().resolve_conj()):  # the lazy one first
        cs, xs = c.detach().requires_grad_(), [v.detach().requires_grad_() for v in x]
        out1 = nb.nufft2d1(*xs, cs, N)
        w = wrap(f)
        out1.backward(w)
        fs, ys = f.detach().requires_grad_(), [v.detach().requires_grad_() for v in x]
        nb.nufft2d2(*ys, fs).backward(wrap(c))
        got = [cs.grad, *[v.grad for v in xs], fs.grad, *[v.grad for v in ys]]
        if w.is_conj():
            lazy = got
    for a, b in zip(lazy, got):
        _close(a, b)


def test_plans():
    x, c, f, _ = _data()
    kp = nb.compute_kernel_params(1e-6)
    ps = PointSort(x, (48, 40), kp, True)
    lazy = PointSort([_neg(v) for v in x], (48, 40), kp, True)
    _close(lazy.spread(c.conj()[None]), ps.spread(c.conj().resolve_conj()[None]))
    fw = ps.spread(c[None])
    _close(ps.interp(fw.conj()), ps.interp(fw.conj().resolve_conj()))
    plan = BatchPlan([[_neg(v) for v in x]], [N])
    f1, c2 = plan.run([c.conj()], [f.conj()])
    _close(f1[0], nb.nufft2d1(*x, c.conj().resolve_conj(), N))
    _close(c2[0], nb.nufft2d2(*x, f.conj().resolve_conj()))
