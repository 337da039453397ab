"""GPU: the 3D gradient pass where bins with fewer points than cells take a lane
group per point and denser bins a thread per point, against the oracle's adjoint
formulas.  Tolerances: complex128 1e-11 (as the other gradient tests); complex64
2e-5, the derivative weights' float error (a few 1e-6) and the footprint sums'."""

import numpy as np
import pytest
import torch

import nufftax_b200 as nb
from nufftax_b200._plan import PointSort
from oracle import nufft_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("eps", [1e-3, 1e-6])
@pytest.mark.parametrize("cdt", [np.complex64, np.complex128])
@pytest.mark.parametrize("kind", ["sparse", "mixed"])
def test_gradient_of_sparse_and_dense_bins(eps, cdt, kind):
    rng = np.random.default_rng(11)
    kp = nb.compute_kernel_params(eps)
    nf, nt = (36, 30, 27), 2
    rdt = np.float32 if cdt == np.complex64 else np.float64
    # "mixed": every point of a narrow cluster falls in a few bins (16 x 16 x 8
    # cells) with more points than cells, the rest in bins with fewer
    M = 37 if kind == "sparse" else 9001
    X = rng.uniform(-np.pi, np.pi, (3, M))
    if kind == "mixed":
        X[:, : 3 * M // 4] = 0.15 * rng.standard_normal((3, 3 * M // 4)) + 0.4
    X = [x.astype(rdt) for x in X]
    c = (rng.standard_normal((nt, M)) + 1j * rng.standard_normal((nt, M))).astype(cdt)
    g = (rng.standard_normal((nt,) + nf[::-1]) + 1j * rng.standard_normal((nt,) + nf[::-1])).astype(cdt)
    dev = torch.device("cuda", 0)
    ps = PointSort([torch.from_numpy(x).to(dev) for x in X], nf, kp, prenorm=False)
    if kind == "mixed":
        counts = np.diff(ps.results()[2].cpu().numpy())
        cells = int(np.prod(ps.tile))
        assert counts.max() >= cells and (counts[counts > 0] < cells).any()
    dc, dxs = ps.spread_grad(torch.from_numpy(c).to(dev), torch.from_numpy(g).to(dev), True, [True] * 3)
    tol = 2e-5 if cdt == np.complex64 else 1e-11
    assert O.rel_l2(dc.cpu().numpy(), O.interp(X, g, kp)) < tol
    ref = O.spread_grad_coords(X, c, g, kp)
    for d in range(3):
        assert O.rel_l2(dxs[d].cpu().numpy(), ref[d]) < tol
    # one output only, and the interpolation's form (no value output)
    only = ps.interp_grad(torch.from_numpy(g).to(dev), torch.from_numpy(c).to(dev), [False, True, False])
    assert only[0] is None and only[2] is None
    assert O.rel_l2(only[1].cpu().numpy(), ref[1]) < tol
