"""FP64 SVD at any scale of the input and beside rows far below the largest: squared norms
and dot products must not leave the range of normal numbers."""

import numpy as np
import pytest
import torch

import acetn_gb300 as gb

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -52


def run(a):
    out = [t.cpu().numpy() for t in gb.svd(torch.from_numpy(np.ascontiguousarray(a)).cuda())]
    assert gb._abi.device_status() == 0
    return out


# the cluster form alone and with the FP32 stage, the Householder and the Cholesky route,
# global memory
@pytest.mark.parametrize("m,n", [(1, 1), (22, 80), (25, 25), (60, 57), (144, 144), (200, 200),
                                 (1500, 90), (480, 470)])
@pytest.mark.parametrize("power", [-960, -520, 500, 1000])
def test_power_of_two(m, n, power):
    """Scaling by a power of two is exact: the same vectors and scaled values, bit for bit."""
    a = np.random.default_rng(m + n).uniform(0.25, 1, (m, n))
    u, s, v = run(a)
    u2, s2, v2 = run(np.ldexp(a, power))
    assert np.array_equal(u, u2) and np.array_equal(v, v2)
    assert np.array_equal(np.ldexp(s, power), s2)


@pytest.mark.parametrize("m,n", [(22, 80), (80, 22), (30, 40)])
@pytest.mark.parametrize("small", [1e-120, 1e-150, 1e-200])
def test_small_rows(m, n, small):
    """Half of the short side's vectors far below the others: rotated among themselves as
    if they stood alone (one-sided Jacobi; the bound of the SVD tests)."""
    rng = np.random.default_rng(1)
    p, length = min(m, n), max(m, n)
    w = rng.standard_normal((p, length))
    w[::2] *= small
    a = w if m < n else w.T
    u, s, v = run(a)
    c = 50 * np.sqrt(length) * EPS
    long_side = v if m < n else u
    assert np.abs(long_side.T @ long_side - np.eye(p)).max() <= c
    top, rest = s[: p // 2], s[p - p // 2:]
    assert np.all(np.diff(s) <= 0) and rest.max() < 1e3 * small < top.min()
    ref = np.linalg.svd(w[1::2], compute_uv=False)
    assert np.abs(top - ref[: len(top)]).max() <= c * top[0]
