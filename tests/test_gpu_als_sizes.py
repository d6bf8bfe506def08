"""The ALS least-squares kernel at the edges of its blocks (systems of 1, 31, 32, 33
and 160 unknowns, 1 to 8 right-hand sides) against the oracle after two iterations.
The systems' condition stays below 1e5, so 1e5 times the rounding unit times m is
2e-9 at most."""

import numpy as np
import pytest
import torch

import acetn_gb300 as gb
from oracle import ctm_oracle as orc

pytestmark = pytest.mark.gpu


class Config:
    als_niter, als_tol, als_method, als_epsilon = 2, 0.0, "cholesky", 1e-12


@pytest.mark.parametrize("shape", [(1, 1, 1), (31, 1, 2), (8, 4, 2), (11, 3, 8), (16, 10, 2),
                                   (20, 8, 8)])
def test_als_sizes(shape):
    nD, bD, pD = shape
    rng = np.random.default_rng(nD * bD + pD)
    n = rng.standard_normal((nD * nD, 2 * nD * nD)) / nD
    n12 = (n @ n.T + 0.5 * np.eye(nD * nD)).reshape(nD, nD, nD, nD)
    a12g = rng.standard_normal((nD, nD, pD, pD))
    g = [torch.from_numpy(x).cuda() for x in (n12, a12g)]
    a1r, a2r = gb.ALSSolver(*g, shape, Config()).solve()
    mine = torch.einsum("yup,xuq->yxpq", a1r, a2r).cpu().numpy()
    b1, b2, _ = orc.als_solve(n12, a12g, shape, niter=2, tol=0.0)
    ref = np.einsum("yup,xuq->yxpq", b1, b2)
    assert np.abs(mine - ref).max() < 2e-9 * np.abs(ref).max()
