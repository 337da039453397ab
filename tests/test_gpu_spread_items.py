"""GPU: the window spread's work items: sizes around the smallest item, whole rounds
of the resident CTAs, and 3D items on both sides of the largest number of blocks that
is grouped, against the oracle.  Tolerances as the window spread's own tests."""

import numpy as np
import pytest
import torch

import nufftax_b200 as nb
from nufftax_b200._plan import PointSort
from oracle import nufft_oracle as O

pytestmark = pytest.mark.gpu

EPS_OF = {2: 1e-1, 4: 1e-3, 6: 1e-5, 8: 1e-6, 14: 1e-12}
C64, C128 = np.complex64, np.complex128
CASES = [
    # dim, nf, ns, M, dtype
    (2, (64, 48), 8, 31, C64),
    (2, (64, 48), 8, 32, C64),
    (2, (64, 48), 8, 33, C64),
    (2, (96, 80), 8, 148 * 4 * 32, C64),      # one item of 32 points for each of four CTAs an SM
    (2, (96, 80), 8, 148 * 4 * 32 + 1, C64),
    (2, (96, 80), 4, 37_888, C64),
    (2, (64, 60), 14, 148 * 32 + 1, C128),
    (2, (64, 60), 14, 33, C128),
    (3, (32, 30, 28), 8, 33, C64),
    (3, (32, 30, 28), 8, 148 * 2 * 32 + 1, C64),
    (3, (32, 30, 28), 4, 5000, C128),
    (3, (160, 160, 128), 8, 330, C64),        # an item spans about 5000 blocks: not grouped
    (3, (160, 160, 128), 6, 500, C64),        # about 3300
    (3, (160, 160, 128), 4, 1700, C64),       # about 1000
]


@pytest.mark.parametrize("case", range(len(CASES)))
def test_items(case):
    dim, nf, ns, M, cdt = CASES[case]
    rng = np.random.default_rng(300 + case)
    kp = nb.compute_kernel_params(EPS_OF[ns])
    assert kp.nspread == ns
    rdt = np.float32 if cdt is C64 else np.float64
    X = [x.astype(rdt) for x in rng.uniform(-np.pi, np.pi, (dim, M))]
    c = (rng.standard_normal((1, M)) + 1j * rng.standard_normal((1, M))).astype(cdt)
    dev = torch.device("cuda", 0)
    ps = PointSort([torch.from_numpy(x).to(dev) for x in X], nf, kp, prenorm=False)
    got = ps.spread(torch.from_numpy(c).to(dev)).cpu().numpy()
    want = O.spread(X, c, nf, kp)
    assert O.rel_l2(got, want) <= (1e-5 if cdt is C64 else 1e-12)
