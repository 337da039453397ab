"""GPU: sorts by 11-bit digits on both sides of their chunk sizes (1024-element chunks
up to 75,776 points, 4096 above), bit-exact against the oracle."""

import numpy as np
import pytest
import torch

import nufftax_b200 as nb
from nufftax_b200._plan import PointSort
from oracle import nufft_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,nf", [(1, (2_097_152,)), (2, (2048, 1944))])
@pytest.mark.parametrize("M,rdt", [(75_775, np.float64), (75_776, np.float32), (75_777, np.float32), (75_777, np.float64)])
def test_sort_around_the_11_bit_chunk_size(dim, nf, M, rdt):
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
