"""GPU: the complex128 ES weights (inner weights by polynomial, edge weights by
exp/sqrt) against extended precision.

One point of unit strength spread on its own 1D grid gives the weights
themselves.  Bound: the fit is accepted within 4e-16 of each weight's largest
value (at most 1); the edge weights by exp/sqrt are off by the rounding of their
exponent, beta (sqrt(..) - 1), relative to the weight: 0.30 at width 4 (beta 9: about
1.1e-15 of it), 0.029 at 6, 1.8e-3 at 8 and less beyond.  So 6e-16 absolute."""

import numpy as np
import pytest
import torch

import nufftax_b200 as nb
from nufftax_b200.core import interp_1d, spread_1d

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("upsampfac", [2.0, 1.25])
@pytest.mark.parametrize("eps", [1e-3, 1e-5, 1e-6, 1e-9, 1e-11, 1e-12, 1e-15])
def test_double_weights_vs_extended_precision(eps, upsampfac):
    kp = nb.compute_kernel_params(eps, upsampfac)
    ns, nf, n = kp.nspread, 64, 65
    rng = np.random.default_rng(3)
    xs = np.concatenate([rng.uniform(-np.pi, np.pi, n - 3), [0.0, np.pi / 3, -2.5]])
    x = torch.from_numpy(xs).cuda()
    # the fold in double, as the kernels round it
    t = xs * (1.0 / (2.0 * np.pi)) + 0.5
    s = (t - np.floor(t)) * nf
    i0 = np.ceil(s - ns / 2).astype(int)
    L = np.longdouble
    want = np.zeros((n, nf))
    for q in range(ns):
        z = (i0 + q).astype(L) - s.astype(L)
        arg = L(1) - L(kp.c) * z * z
        w = np.where(arg >= 0, np.exp(L(kp.beta) * (np.sqrt(np.maximum(arg, L(0))) - L(1))), L(0))
        want[np.arange(n), (i0 + q) % nf] = w.astype(np.float64)
    for j in range(n):
        fw = spread_1d(x[j:j + 1], torch.ones(1, dtype=torch.complex128, device="cuda"), nf, kp).cpu().numpy()
        assert np.max(np.abs(fw.real - want[j])) < 6e-16
    # the interpolation reads the same weights back, one grid cell at a time
    e = torch.zeros(nf, dtype=torch.complex128, device="cuda")
    e[10] = 1.0
    got = interp_1d(x, e, nf, kp).cpu().numpy().real
    assert np.max(np.abs(got - want[:, 10])) < 6e-16
