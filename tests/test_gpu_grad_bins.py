"""GPU: the 3D gradient pass at the bin sizes where its form changes (a lane group per
point from 128 points up to the tile's cells, else a thread per point), against the
oracle's adjoint formulas.  Tolerances as the lane-group gradient's own test."""

import numpy as np
import pytest
import torch

import nufftax_b200 as nb
from nufftax_b200._plan import PointSort
from oracle import nufft_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cdt", [np.complex64, np.complex128])
@pytest.mark.parametrize("eps", [1e-3, 1e-6])
def test_gradient_at_the_edges_of_its_bin_rule(eps, cdt):
    rng = np.random.default_rng(17)
    kp = nb.compute_kernel_params(eps)
    nf, counts = (48, 32, 16), [1, 127, 128, 129, 2047, 2048]
    dev = torch.device("cuda", 0)
    rdt = np.float32 if cdt == np.complex64 else np.float64
    tile = PointSort([torch.zeros(1, dtype=torch.float32 if rdt is np.float32 else torch.float64, device=dev)] * 3, nf,
                     kp, prenorm=False).tile
    nb_axis = [n // t for n, t in zip(nf, tile)]
    # bin b's points: left cells inside the tile, off its edges
    X = []
    for b, n in enumerate(counts):
        o = [b % nb_axis[0] * tile[0], b // nb_axis[0] % nb_axis[1] * tile[1], b // (nb_axis[0] * nb_axis[1]) * tile[2]]
        X.append([(o[d] + (tile[d] - 1.2) * rng.random(n) + 0.1 + kp.nspread / 2) / nf[d] for d in range(3)])
    X = [np.concatenate([x[d] for x in X]) for d in range(3)]
    X = [((np.mod(x, 1.0) - 0.5) * 2 * np.pi).astype(rdt) for x in X]
    M = X[0].size
    c = (rng.standard_normal((1, M)) + 1j * rng.standard_normal((1, M))).astype(cdt)
    g = (rng.standard_normal((1,) + nf[::-1]) + 1j * rng.standard_normal((1,) + nf[::-1])).astype(cdt)
    ps = PointSort([torch.from_numpy(x).to(dev) for x in X], nf, kp, prenorm=False)
    got_counts = np.diff(ps.results()[2].cpu().numpy())
    assert sorted(got_counts[got_counts > 0]) == counts and int(np.prod(ps.tile)) == 2048
    dc, dxs = ps.spread_grad(torch.from_numpy(c).to(dev), torch.from_numpy(g).to(dev), True, [True] * 3)
    tol = 2e-5 if cdt == np.complex64 else 1e-11
    assert O.rel_l2(dc.cpu().numpy(), O.interp(X, g, kp)) < tol
    ref = O.spread_grad_coords(X, c, g, kp)
    for d in range(3):
        assert O.rel_l2(dxs[d].cpu().numpy(), ref[d]) < tol
