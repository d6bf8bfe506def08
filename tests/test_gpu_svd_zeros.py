"""FP64 SVD of matrices with singular values that are exactly zero (padding, a zero matrix),
through the QR routes: the short side's vectors are an orthonormal basis all the same
(bound of the SVD tests)."""

import numpy as np
import pytest
import torch

import acetn_gb300 as gb

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -52


@pytest.mark.parametrize("m,n", [(40, 40), (33, 60), (60, 33), (144, 144), (149, 180), (90, 1500)])
@pytest.mark.parametrize("rank", [0, 1, 0.5, -1])
def test_orthonormal_short_side(m, n, rank):
    rng = np.random.default_rng(m + n)
    p = min(m, n)
    r = rank if rank in (0, 1) else int(p * rank) if rank > 0 else p + rank
    a = np.zeros((m, n))
    rows, cols = rng.permutation(m)[:r], rng.permutation(n)[:r]
    a[np.ix_(rows, cols)] = rng.standard_normal((r, r))
    u, s, v = (t.cpu().numpy() for t in gb.svd(torch.from_numpy(a).cuda()))
    assert gb._abi.device_status() == 0
    c = 50 * np.sqrt(max(m, n)) * EPS
    short = u if m <= n else v
    assert np.abs(short.T @ short - np.eye(p)).max() <= c
    assert np.linalg.norm((u * s) @ v.T - a, 2) <= c * max(1.0, np.abs(s).max())
    assert np.all(s[r:] <= c * max(1.0, s[0]))


@pytest.mark.parametrize("m,n", [(60, 1200), (470, 460)])
def test_global_memory_form(m, n):
    """Rank-deficient ones that the Cholesky route leaves to it, and large ones: rows that
    collapse end as zeros within the sweep limit."""
    rng = np.random.default_rng(m)
    a = np.zeros((m, n))
    a[: m // 2] = rng.standard_normal((m // 2, n))
    a[m // 2: m - 3] = rng.standard_normal((m - 3 - m // 2, m // 2)) @ a[: m // 2]
    u, s, v = (t.cpu().numpy() for t in gb.svd(torch.from_numpy(a).cuda()))
    assert gb._abi.device_status() == 0
    c = 50 * np.sqrt(max(m, n)) * EPS
    short = u if m <= n else v
    assert np.abs(short.T @ short - np.eye(min(m, n))).max() <= c
    assert np.linalg.norm((u * s) @ v.T - a, 2) <= c * s[0]
    assert np.all(s[m // 2:] <= c * s[0])
