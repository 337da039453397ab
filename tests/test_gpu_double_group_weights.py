"""GPU: complex128 weights of the interpolations with a lane group per point (3D, and
2D on request) and with a thread per point (2D), read back from single grid cells
against extended precision.

Bound: each axis' weight, at most 1, is off by the rounding of its exponent
beta (sqrt(1 - c z^2) - 1), at most (1.2 beta + 4) 2^-53 (sqrt and its argument, the
product, exp); a product of dim weights by dim times that."""

import numpy as np
import pytest
import torch

import nufftax_b200 as nb
from nufftax_b200._plan import PointSort

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,mode", [(2, 0), (2, 2), (3, 0)])  # 2: a lane group per point
@pytest.mark.parametrize("eps", [1e-3, 1e-5, 1e-6, 1e-9, 1e-12])
def test_interpolation_weights(eps, dim, mode):
    kp = nb.compute_kernel_params(eps)
    ns, nf, n = kp.nspread, (40, 36, 34)[:dim], 400
    rng = np.random.default_rng(5)
    L = np.longdouble
    X, W, cell = [], np.ones(n, dtype=L), []
    for d in range(dim):
        # points around one cell, so that most footprints hold it
        x = (rng.uniform(17 - ns / 2, 17 + ns / 2, n) / nf[d] - 0.5) * 2 * np.pi
        t = x * (1.0 / (2.0 * np.pi)) + 0.5  # the fold in double, as the kernels round it
        s = (t - np.floor(t)) * nf[d]
        z = L(17) - s.astype(L)
        arg = L(1) - L(kp.c) * z * z
        inside = (17 >= np.ceil(s - ns / 2)) & (17 < np.ceil(s - ns / 2) + ns)
        W *= np.where((arg >= 0) & inside, np.exp(L(kp.beta) * (np.sqrt(np.maximum(arg, L(0))) - L(1))), L(0))
        X.append(x)
        cell.append(17)
    dev = torch.device("cuda", 0)
    ps = PointSort([torch.from_numpy(x).to(dev) for x in X], nf, kp, prenorm=False, modes=(0, mode))
    fw = torch.zeros((1,) + nf[::-1], dtype=torch.complex128, device=dev)
    fw[(0,) + tuple(cell)] = 1.0
    got = ps.interp(fw).cpu().numpy()[0]
    assert np.max(np.abs(got.real - W.astype(np.float64))) <= dim * (1.2 * kp.beta + 4) * 2.0**-53
    assert np.all(got.imag == 0)
