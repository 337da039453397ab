"""GPU: the register-window spread (2D, 3D widths up to 8) at the edges of its
work items, blocks and windows, against the oracle.

Tolerances: complex128 1e-12 (the sums' rounding, a few hundred terms); complex64
1e-5, the weights' float error (about 1e-6) and the sums' with a margin, as the
other float spreads' tests."""

import numpy as np
import pytest
import torch

import nufftax_b200 as nb
from nufftax_b200._plan import PointSort
from oracle import nufft_oracle as O

pytestmark = pytest.mark.gpu

EPS_OF = {2: 1e-1, 4: 1e-3, 6: 1e-5, 8: 1e-6, 14: 1e-12, 16: 1e-15}


def _spread(X, c, nf, kp, modes=(0, 0)):
    dev = torch.device("cuda", 0)
    ps = PointSort([torch.from_numpy(x).to(dev) for x in X], nf, kp, prenorm=False, modes=modes)
    return ps.spread(torch.from_numpy(c).to(dev)).cpu().numpy()


def _points(rng, dim, M, kind, rdt):
    if kind == "uniform":
        X = rng.uniform(-np.pi, np.pi, (dim, M))
    elif kind == "clustered":
        X = np.mod(0.02 * rng.standard_normal((dim, M)) + np.pi, 2 * np.pi) - np.pi
    else:  # "edge": around the periodic boundary, every window wraps
        X = np.mod(np.pi + 0.05 * rng.standard_normal((dim, M)) + np.pi, 2 * np.pi) - np.pi
    return [x.astype(rdt) for x in X]


CASES = [
    # dim, nf, ns, M, n_trans, dtype, points
    (2, (64, 48), 8, 1, 1, np.complex64, "uniform"),
    (2, (64, 48), 8, 33, 2, np.complex64, "edge"),
    (2, (45, 27), 6, 1001, 1, np.complex64, "uniform"),        # odd grid rows
    (2, (300, 200), 4, 40_000, 1, np.complex64, "clustered"),  # items of 512 points
    (2, (16, 16), 8, 700, 3, np.complex64, "uniform"),         # the window covers the grid
    (2, (40, 36), 2, 500, 1, np.complex64, "edge"),
    (2, (64, 60), 14, 2500, 2, np.complex128, "uniform"),
    (2, (90, 70), 16, 300, 1, np.complex128, "edge"),
    (2, (160, 160), 8, 38_001, 1, np.complex128, "clustered"),
    (3, (32, 30, 27), 8, 1, 1, np.complex64, "uniform"),
    (3, (32, 30, 27), 8, 2049, 2, np.complex64, "edge"),
    (3, (160, 160, 128), 8, 700, 1, np.complex64, "uniform"),  # too few points per bin to group
    (3, (16, 18, 20), 8, 5000, 1, np.complex64, "clustered"),  # the window nearly covers the grid
    (3, (40, 44, 48), 6, 40_000, 1, np.complex64, "uniform"),
    (3, (33, 35, 31), 4, 3000, 2, np.complex64, "uniform"),
    (3, (20, 22, 24), 2, 400, 1, np.complex128, "uniform"),
    (3, (24, 20, 22), 6, 3000, 1, np.complex128, "edge"),
    (3, (20, 20, 20), 8, 9000, 2, np.complex128, "uniform"),   # denser than cells
]


@pytest.mark.parametrize("case", range(len(CASES)))
def test_window_spread_vs_oracle(case):
    dim, nf, ns, M, nt, cdt, kind = CASES[case]
    rng = np.random.default_rng(100 + case)
    kp = nb.compute_kernel_params(EPS_OF[ns])
    assert kp.nspread == ns
    rdt = np.float32 if cdt == np.complex64 else np.float64
    X = _points(rng, dim, M, kind, rdt)
    c = (rng.standard_normal((nt, M)) + 1j * rng.standard_normal((nt, M))).astype(cdt)
    fw = _spread(X, c, nf, kp, modes=(3, 0))  # a warp per point: the window at every density
    ref = np.stack([O.spread(X, c[t], nf, kp) for t in range(nt)])
    tol = 1e-5 if cdt == np.complex64 else 1e-12
    assert O.rel_l2(fw, ref) < tol


@pytest.mark.parametrize("dim,cdt", [(2, np.complex64), (2, np.complex128), (3, np.complex64)])
def test_non_finite_strengths_stay_in_their_footprints(dim, cdt):
    """An infinite or NaN strength reaches exactly its own footprint's cells: the
    zero weights of the rest of its window do not turn into NaN."""
    rng = np.random.default_rng(5)
    nf = (48, 40) if dim == 2 else (32, 28, 24)
    kp = nb.compute_kernel_params(1e-6)
    rdt = np.float32 if cdt == np.complex64 else np.float64
    M = 200
    X = _points(rng, dim, M, "uniform", rdt)
    c = (rng.standard_normal((1, M)) + 1j * rng.standard_normal((1, M))).astype(cdt)
    clean = c.copy()
    bad = [17, 101]
    clean[0, bad] = 0
    c[0, 17] = np.inf
    c[0, 101] = complex(np.nan, 1.0)
    fw = _spread(X, c, nf, kp, modes=(3, 0))[0]
    one = np.zeros((1, M), cdt)
    one[0, bad] = 1
    touched = _spread(X, one, nf, kp, modes=(3, 0))[0] != 0
    assert np.array_equal(~np.isfinite(fw), touched)
    ref = O.spread(X, clean[0], nf, kp)
    tol = 1e-5 if cdt == np.complex64 else 1e-12
    assert O.rel_l2(fw[~touched], ref[~touched]) < tol
