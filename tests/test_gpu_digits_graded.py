"""FP64 digit products of rows and columns whose large entries do not meet: every output
as close to the exact one as an FMA chain's, beside sum_k |a_k b_k| and not beside the
product of the two rows' largest entries.

Bar: where the digits stand, that sum is at least 2^-8.4 of the scales' product, and the
dropped digit products deviate by sqrt(K) 2^-62.2 of it (the streaming form's rounding by
2^-59.8 to 2^-57.8 besides, K >= 16 to 81): sqrt(K) 2^-53 of the sum at most.  Six
deviations and the last rounding are below 8 sqrt(K) 2^-53; a chain of K FMAs is too."""

import numpy as np
import pytest
import torch

import acetn_gb300 as gb
from test_gpu_digits import product, run

pytestmark = pytest.mark.gpu

# column tiles, K ranges, ranges summed apart, the streaming form (one and two phases, on
# either side, the three groups of K)
SHAPES = [(700, 400, 100), (5000, 300, 40), (385, 259, 256), (128, 64, 2881), (19, 300, 70001),
          (9000, 100, 150), (30000, 24, 30), (36, 9001, 72), (8200, 60, 45)]


def check(a, b):
    c = run(a, b)
    i = np.unique(np.linspace(0, a.shape[0] - 1, 60).astype(int))
    j = np.unique(np.linspace(0, b.shape[1] - 1, 60).astype(int))
    a, b, c = a[i], b[:, j], c[np.ix_(i, j)]
    bar = 8 * a.shape[1] ** 0.5 * 2.0 ** -53 * (np.abs(a) @ np.abs(b))
    err = np.abs((c - product(a, b)).astype(float))
    assert np.all(err <= bar), float((err / np.maximum(bar, 1e-300)).max())


def normals(m, n, k, seed):
    rng = np.random.default_rng(seed)
    return rng.standard_normal((m, k)), rng.standard_normal((k, n)), rng


@pytest.mark.parametrize("m,n,k", SHAPES)
@pytest.mark.parametrize("bits", [20, 60, 400])
def test_opposed(m, n, k, bits):
    a, b, _ = normals(m, n, k, bits)
    s = 2.0 ** -np.round(bits * np.arange(k) / k)
    check(a * s, b / s[:, None])


@pytest.mark.parametrize("m,n,k", SHAPES)
def test_each_row_its_own_way(m, n, k):
    """Half of the rows graded down, half up, columns at random: no scaling of the
    contracted index helps.  One row of one entry, columns without some or all of them."""
    a, b, rng = normals(m, n, k, 7)
    t = np.arange(k) / k
    up = rng.random(m) < 0.5
    a *= 2.0 ** (-40 * np.where(up[:, None], t, 1 - t))
    b *= 2.0 ** (-40 * np.abs(t[:, None] - rng.random(n)))
    a[m // 2] = 0.0
    a[m // 2, k // 3] = 3.0
    b[k // 3, :n // 2] = 0.0
    b[:, 1] = 0.0
    b[k // 3, 2] = 1e-300
    check(a, b)


@pytest.mark.parametrize("m,n,k", [(700, 400, 100), (128, 64, 2881), (9000, 100, 150), (30000, 24, 30)])
def test_blocks(m, n, k):
    """Two blocks without common indices: zeros outside them, exactly."""
    a, b, _ = normals(m, n, k, 9)
    a[: m // 2, k // 2:] = 0.0
    a[m // 2:, : k // 2] = 0.0
    b[k // 2:, : n // 3] = 0.0
    b[: k // 2, n // 3:] = 0.0
    c = run(a, b)
    assert not c[: m // 2, n // 3:].any() and not c[m // 2:, : n // 3].any()
    check(a, b)


def test_kept_digits():
    """A randomized SVD keeps its factors' digits: the singular values of a product whose
    inner legs are graded by 2^-40 and 2^40 (well-conditioned in exact arithmetic)."""
    rng = np.random.default_rng(3)
    m, k = 1600, 128
    a, b = rng.standard_normal((m, k)), rng.standard_normal((k, m))
    want = np.linalg.svd(a @ b, compute_uv=False)[:k]
    s = 2.0 ** -np.round(40 * np.arange(k) / k)
    got = gb.fused_matmul_svd_lowrank(torch.from_numpy(a * s).cuda(),
                                      torch.from_numpy(b / s[:, None]).cuda(), q=k, niter=1)[1]
    assert gb._abi.device_status() == 0
    assert np.abs(got.cpu().numpy() - want).max() < 1e-12 * want[0]


@pytest.mark.parametrize("bits", [0, 40, 300])
def test_qr_of_graded_columns(bits):
    """Columns of norms from 1 to 2^-bits: the residual beside each column's norm (bound of
    the Cholesky-QR tests, 20 sqrt(n q) eps), whose factor L^-1 is graded the other way."""
    rng = np.random.default_rng(11)
    n, q = 1700, 132
    a = rng.standard_normal((n, q)) * 2.0 ** -np.round(bits * np.arange(q) / q)
    gb._abi.qr_fallbacks()  # (a query resets the count)
    qm, r = (t.cpu().numpy() for t in gb.qr(torch.from_numpy(a).cuda()))
    assert gb._abi.qr_fallbacks() == 0
    c = 20 * np.sqrt(n * q) * 2.0 ** -52
    assert np.abs(qm.T @ qm - np.eye(q)).max() <= c
    assert np.all(np.linalg.norm(qm @ r - a, axis=0) <= c * np.linalg.norm(a, axis=0))
    assert np.array_equal(r, np.triu(r)) and np.all(np.diag(r) > 0)
