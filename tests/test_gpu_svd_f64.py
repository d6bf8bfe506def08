"""FP64 thin SVD at the edges of its cluster shapes, of the reduction to a
triangular factor and of the global-memory form, against LAPACK.

Bounds: one-sided Jacobi and the Cholesky-QR are backward stable, so the
residual and the singular values are within c eps |A| and the vectors
orthonormal to c eps; c = 50 sqrt(max(m, n)) covers the accumulated roundings
of 15 sweeps (each entry takes about 15 max(m, n) rotations of 3 roundings,
which add up like a random walk)."""

import numpy as np
import pytest
import torch

import acetn_gb300 as gb

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -52


def matrix(m, n, kind, seed=0):
    rng = np.random.default_rng(seed + 1000 * m + n)
    a = rng.standard_normal((m, n))
    r = min(m, n)
    if kind == "graded":  # singular values from 1 down to 1e-13
        u, v = np.linalg.qr(rng.standard_normal((m, r)))[0], np.linalg.qr(rng.standard_normal((n, r)))[0]
        a = (u * 10.0 ** (-13 * np.arange(r) / max(1, r - 1))) @ v.T
    elif kind == "deficient":
        a = a[:, : max(1, r // 3)] @ rng.standard_normal((max(1, r // 3), n))
    elif kind == "equal":  # all singular values equal
        a = np.linalg.qr(rng.standard_normal((max(m, n), r)))[0]
        a = a if m >= n else a.T
    return np.ascontiguousarray(a)


SHAPES = [(1, 1), (2, 1), (1, 5), (2, 2), (3, 3), (4, 7), (5, 4), (17, 17), (22, 80), (33, 32),
          (48, 31), (66, 66), (127, 128), (144, 144), (161, 160), (290, 289), (462, 150),
          # reduced to the triangular factor (long side > 6 x short side)
          (66, 1024), (1500, 90), (161, 1900),
          # too large for the cluster
          (480, 470)]


def check(a, u, s, v):
    m, n = a.shape
    r = min(m, n)
    top = np.abs(s).max()
    c = 50 * np.sqrt(max(m, n)) * EPS
    ref = np.linalg.svd(a, compute_uv=False)
    assert u.shape == (m, r) and s.shape == (r,) and v.shape == (n, r)
    assert np.all(np.diff(s) <= 0) and np.abs(s - ref).max() <= c * top
    assert np.linalg.norm((u * s) @ v.T - a, 2) <= c * top
    return c


@pytest.mark.parametrize("m,n", SHAPES)
@pytest.mark.parametrize("kind", ["random", "graded", "equal"])
def test_svd_shapes(m, n, kind):
    if kind != "random" and max(m, n) > 1000 and min(m, n) > 100:
        pytest.skip("covered by the smaller shapes")
    a = matrix(m, n, kind)
    u, s, v = (t.cpu().numpy() for t in gb.svd(torch.from_numpy(a).cuda()))
    c = check(a, u, s, v)
    if (m, n) != (480, 470) or kind == "random":  # graded rows take the grid form 20 sweeps
        for w in (u, v):
            # vectors of singular values at the rounding level of the largest are
            # normalised rounding errors
            w = w[:, s > 1e-9 * s[0]]
            assert np.abs(w.T @ w - np.eye(w.shape[1])).max() <= c
    assert gb._abi.device_status() == 0


@pytest.mark.parametrize("m,n", [(40, 40), (60, 1200), (1201, 61)])
def test_svd_rank_deficient(m, n):
    a = matrix(m, n, "deficient")
    u, s, v = (t.cpu().numpy() for t in gb.svd(torch.from_numpy(a).cuda()))
    check(a, u, s, v)
    assert np.isfinite(u).all() and np.isfinite(v).all()
    z = gb.svd(torch.zeros(m, n, dtype=torch.float64, device="cuda"))
    assert all(bool(torch.isfinite(t).all()) for t in z) and float(z[1].abs().max()) == 0.0
    assert gb._abi.device_status() == 0
