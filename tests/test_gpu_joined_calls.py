"""GPU: the joined native calls (spread + FFT + deconvolution; deconvolution + FFT)
against the same steps one by one, and transforms that alternate through more shapes
and point counts than the library keeps resolved per thread.  The spread's atomics
order float sums differently from run to run: 1e-6 for complex64, 1e-14 for complex128."""

import pytest
import torch

import nufftax_b200 as nb
from nufftax_b200 import profiling

pytestmark = pytest.mark.gpu

T1 = {1: nb.nufft1d1, 2: nb.nufft2d1, 3: nb.nufft3d1}
T2 = {1: nb.nufft1d2, 2: nb.nufft2d2, 3: nb.nufft3d2}


def _case(dim, M, n, cdt, seed, nt=2):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    rdt = torch.float32 if cdt == torch.complex64 else torch.float64
    x = [(torch.rand(M, generator=g, device="cuda", dtype=rdt) * 2 - 1) * 3.1 for _ in range(dim)]
    c = torch.randn((nt, M), generator=g, device="cuda", dtype=cdt)
    f = torch.randn((nt,) + n[::-1], generator=g, device="cuda", dtype=cdt)
    return x, c, f


def _close(a, b, tol):
    assert torch.linalg.norm(a - b) <= tol * torch.linalg.norm(b)


@pytest.mark.parametrize("cdt,tol", [(torch.complex64, 1e-6), (torch.complex128, 1e-14)])
@pytest.mark.parametrize("dim,n", [(1, (50,)), (2, (24, 31)), (3, (12, 9, 14))])
def test_joined_calls_equal_their_steps(dim, n, cdt, tol):
    x, c, f = _case(dim, 900, n, cdt, dim)
    nn = n if dim > 1 else n[0]
    f1, c2 = T1[dim](*x, c, nn), T2[dim](*x, f)
    with profiling.record() as rec:  # call by call
        f1s, c2s = T1[dim](*x, c, nn), T2[dim](*x, f)
    names = set(rec.summary())
    assert {"nfx_spread_sorted", "nfx_fft", "nfx_deconv_shuffle", "nfx_deconv_pad", "nfx_interp_sorted"} <= names
    _close(f1, f1s, tol)
    _close(c2, c2s, tol)


def test_many_shapes_in_turn():
    cases = [(2, 100 + 37 * k, (16 + 2 * (k % 5), 20 + k % 3)) for k in range(14)]
    first = []
    for rnd in range(2):
        for k, (dim, M, n) in enumerate(cases):
            x, c, f = _case(dim, M, n, torch.complex128, 50 + k)
            nb.sort_cache.clear()
            out = T1[dim](*x, c, n), T2[dim](*x, f)
            if rnd == 0:
                first.append(out)
                # <type 1 (c), f> = <c, type 2 with the opposite sign (f)>
                back = T2[dim](*x, f, isign=-1)
                a, b = (out[0] * f.conj()).sum(), (c * back.conj()).sum()
                assert abs(a - b) <= 1e-4 * (out[0].norm() * f.norm())
            else:
                for u, v in zip(out, first[k]):
                    _close(u, v, 1e-14)
