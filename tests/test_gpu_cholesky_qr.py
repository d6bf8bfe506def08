"""FP64 Cholesky-QR of tall matrices (the route above n q^2 = 4e6) at the edges of
the factorisation's blocks of eight rows and of its shares of a cluster.

Three Cholesky-QR stages are backward stable and orthonormal to working precision
for conditions up to about 1e12; the bound is that of the Householder tests,
20 sqrt(n q) eps."""

import numpy as np
import pytest
import torch

import acetn_gb300 as gb

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -52


@pytest.mark.parametrize("q", [15, 16, 17, 31, 63, 64, 65, 66, 72, 80, 95, 97, 104, 128, 129, 160,
                               161, 192, 200, 256, 257, 300, 320, 330])
@pytest.mark.parametrize("cond", [1.0, 1e10])
def test_orthonormal_and_upper(q, cond):
    n = int(4.0e6 / q / q) + 2 * q
    assert n * q * q > 4.0e6
    rng = np.random.default_rng(q)
    a = rng.standard_normal((n, q))
    if cond > 1:
        a = (a * 10.0 ** -np.linspace(0, np.log10(cond), q)) @ np.linalg.qr(
            rng.standard_normal((q, q)))[0]
    before = gb._abi.qr_fallbacks()
    qm, r = (t.cpu().numpy() for t in gb.qr(torch.from_numpy(a).cuda()))
    assert gb._abi.qr_fallbacks() == 0 and before >= 0  # the Cholesky route's own result
    c = 20 * np.sqrt(n * q) * EPS
    assert np.abs(qm.T @ qm - np.eye(q)).max() <= c
    assert np.linalg.norm(qm @ r - a, 2) <= c * np.linalg.norm(a, 2)
    assert np.array_equal(r, np.triu(r)) and np.all(np.diag(r) > 0)


def test_rank_deficient_input():
    g = torch.Generator(device="cuda").manual_seed(4)
    a = torch.randn(3000, 50, generator=g, dtype=torch.float64, device="cuda")
    a[:, 30:] = a[:, :20]  # exactly rank deficient: orthonormal with or without the fallback
    qm, r = gb.qr(a)
    eye = torch.eye(50, dtype=torch.float64, device="cuda")
    assert float((qm.T @ qm - eye).abs().max()) < 1e-12
    assert float((qm @ r - a).norm()) < 1e-12 * float(a.norm())
