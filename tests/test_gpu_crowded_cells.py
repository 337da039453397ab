"""GPU: float rounding of the spread where very many points share a cell.

All points lie in one cell, strengths are standard normal, the reference is the
same sum in 64 bits with the float coordinates.  The error of each grid cell is
taken relative to the root of the sum of its squared terms (the size of a sum of
random signs).  The bounds come from a replay on the CPU of float sums in the
order of a shared-memory tile (subproblems of 1024 to 4096 points, eight warps
with two sums each, then one addition to the grid per subproblem): 2.2e-7, 5.3e-7
and 3.3e-7 for 100 k, 1 M and 4 M points in 2D; a plane owner's 2048 points one
after another 8.8e-7 for 1 M in 3D.  Twice that, since the 64 cells of a footprint
share their strengths, plus 1e-7 for the weights' own error (below 2.6e-7 a point,
of either sign).  Slices of a warp added to the grid one by one (64 to 128 points)
have 6.7e-7, 2.1e-6 and 2.3e-6 in the same replay."""

import numpy as np
import pytest
import torch

import nufftax_b200 as nb
from nufftax_b200._plan import PointSort
from oracle import nufft_oracle as O

pytestmark = pytest.mark.gpu

EPS_OF = {4: 1e-3, 6: 1e-5, 8: 1e-6}
NT = 4
CASES = [  # dim, nf, ns, M, replay error
    (2, (256, 192), 8, 100_000, 2.2e-7),
    (2, (256, 192), 8, 1_000_000, 5.3e-7),
    (2, (256, 192), 8, 4_000_000, 3.3e-7),
    (2, (256, 192), 6, 1_000_000, 5.3e-7),
    (2, (256, 192), 4, 20_011, 2.2e-7),   # items of 64 points, one group
    (3, (64, 48, 40), 8, 1_000_000, 8.8e-7),
    (3, (64, 48, 40), 4, 30_007, 8.8e-7),
]


@pytest.mark.parametrize("rdt", [np.float32, np.float64])
@pytest.mark.parametrize("case", range(len(CASES)))
def test_one_crowded_cell(case, rdt):
    dim, nf, ns, M, replay = CASES[case]
    if rdt is np.float64 and M > 100_000:
        M = 100_000
    rng = np.random.default_rng(100 + case)
    kp = nb.compute_kernel_params(EPS_OF[ns])
    assert kp.nspread == ns
    cell = [n // 2 + 3 for n in nf]
    X = [((k - 0.95 + 0.9 * rng.random(M)) * 2 * np.pi / n - np.pi).astype(rdt) for k, n in zip(cell, nf)]
    cdt = np.complex64 if rdt is np.float32 else np.complex128
    c = (rng.standard_normal((NT, M)) + 1j * rng.standard_normal((NT, M))).astype(cdt)
    # 64-bit weights of the folded coordinates
    W, I = [], []
    for x, n in zip(X, nf):
        xs = O.fold_rescale(x, n)
        i0 = np.unique(np.asarray(O.cell_index(xs, ns)))
        assert i0.size == 1
        idx = int(i0[0]) + np.arange(ns)
        W.append(O.es_kernel(idx[None, :] - xs.astype(np.float64)[:, None], kp.beta, kp.c))
        I.append(np.mod(idx, n))
    Wr = W[1] if dim == 2 else (W[2][:, :, None] * W[1][:, None, :]).reshape(M, -1)  # rows (z, y)
    want = np.stack([(Wr * ct[:, None].astype(np.complex128)).T @ W[0] for ct in c])
    size = np.sqrt(np.stack([(Wr**2 * np.abs(ct[:, None].astype(np.complex128))**2).T @ W[0]**2 for ct in c]))

    dev = torch.device("cuda", 0)
    ps = PointSort([torch.from_numpy(x).to(dev) for x in X], nf, kp, prenorm=False)
    got = ps.spread(torch.from_numpy(c).to(dev)).cpu().numpy()
    rows = np.ix_(range(NT), I[1], I[0]) if dim == 2 else np.ix_(range(NT), I[2], I[1], I[0])
    got = got[rows].reshape(want.shape)
    # edge cells' weights may be zero or tiny: their errors count by the largest size
    err = np.sqrt((np.abs(got - want) ** 2).sum() / (size**2).sum())
    assert err <= (2 * replay + 1e-7 if rdt is np.float32 else 1e-13), err
