"""GPU: the sort on both sides of its chunk sizes (1024-element chunks up to
303,104 points, 4096 above), bit-exact against the oracle, and the type-3 target
factor with an odd and an even number of quadrature nodes."""

import numpy as np
import pytest
import torch

import nufftax_b200 as nb
from nufftax_b200._plan import PointSort
from oracle import nufft_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,nf", [(1, (16384,)), (2, (512, 486)), (3, (96, 90, 64))])
@pytest.mark.parametrize("M,rdt", [(1, np.float32), (1023, np.float32), (1025, np.float32), (1025, np.float64),
                                   (303_104, np.float32), (303_104, np.float64), (303_105, np.float32)])
def test_sort_around_chunk_sizes(dim, nf, M, rdt):
    rng = np.random.default_rng(M + dim)
    kp = nb.compute_kernel_params(1e-6)
    X = [x.astype(rdt) for x in rng.uniform(-np.pi, np.pi, (dim, M))]
    ps = PointSort([torch.from_numpy(x).cuda() for x in X], nf, kp, prenorm=True)
    keys, perm, bs = (t.cpu().numpy() for t in ps.results())
    okeys, ocells = O.bin_keys(X, nf, kp.nspread, ps.tile, True)
    nbins = int(np.prod([-(-n // t) for n, t in zip(nf, ps.tile)]))
    operm, obs = O.bin_sort(okeys, ocells, nbins, int(np.prod(ps.tile)))
    assert np.array_equal(keys, okeys)
    assert np.array_equal(perm, operm)
    assert np.array_equal(bs, obs)


@pytest.mark.parametrize("eps", [1e-6, 1e-9, 1e-12])  # 20, 20 and 25 nodes
def test_type3_factor_node_counts(eps):
    """complex128 type 3 against the oracle: 2 eps, or the double rounding of its
    sums (1e-13) where that is more."""
    rng = np.random.default_rng(7)
    M, K = 300, 257
    x, s = rng.uniform(-2.0, 2.0, M), rng.uniform(-25.0, 25.0, K)
    c = rng.standard_normal(M) + 1j * rng.standard_normal(M)
    n = nb.compute_type3_grid_size(x, s, eps=eps)
    got = nb.nufft1d3(*[torch.from_numpy(a).cuda() for a in (x, c, s)], n, eps=eps).cpu().numpy()
    ref = O.nufft_type3([x], c, [s], (n,), eps=eps, isign=1)
    assert O.rel_l2(got, ref) < max(2 * eps, 1e-13)
