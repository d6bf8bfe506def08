"""FP64 Householder QR in a cluster at the edges of its row and column shares,
against LAPACK (same sign convention, so Q and R are compared entry by entry
where the matrix is well conditioned).

Bounds: Householder QR is backward stable with a constant of about
q sqrt(q) in the worst case; on these matrices the roundings of q reflections
of n entries add up like a random walk, 20 sqrt(n q) eps."""

import numpy as np
import pytest
import torch

import acetn_gb300 as gb

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -52
SHAPES = [(1, 1), (2, 1), (2, 2), (3, 2), (7, 7), (8, 3), (31, 31), (33, 32), (34, 33), (80, 22),
          (96, 64), (97, 65), (100, 97), (129, 127), (150, 141), (300, 34), (405, 47), (500, 89),
          (1700, 48), (9000, 5), (40000, 10)]


@pytest.mark.parametrize("n,q", SHAPES)
def test_qr_matches_lapack(n, q):
    assert float(n) * q * q <= 4.0e6  # the small-matrix route
    rng = np.random.default_rng(n + 7 * q)
    a = rng.standard_normal((n, q)) * 10.0 ** rng.uniform(-3, 3, q)
    qm, r = (t.cpu().numpy() for t in gb.qr(torch.from_numpy(a).cuda()))
    c = 20 * np.sqrt(n * q) * EPS
    assert np.abs(qm.T @ qm - np.eye(q)).max() <= c
    assert np.all(np.linalg.norm(qm @ r - a, axis=0) <= c * np.linalg.norm(a, axis=0))
    assert np.array_equal(r, np.triu(r))
    q0, r0 = np.linalg.qr(a)
    if n == q:  # LAPACK leaves the last entry as it is, this QR reflects it
        flip = -np.sign(r0[-1, -1] * r[-1, -1])
        q0[:, -1], r0[-1] = -flip * q0[:, -1], -flip * r0[-1]
    assert np.array_equal(np.sign(np.diag(r)), np.sign(np.diag(r0)))
    cond = np.linalg.cond(a / np.linalg.norm(a, axis=0))
    assert np.abs(qm - q0).max() <= 2 * c * cond


@pytest.mark.parametrize("kind", ["deficient", "graded", "zero", "tiny", "huge"])
def test_qr_any_rank_and_scale(kind):
    rng = np.random.default_rng(11)
    a = rng.standard_normal((211, 43))
    if kind == "deficient":
        a = a[:, :5] @ rng.standard_normal((5, 43))
    elif kind == "graded":
        a *= 10.0 ** -np.linspace(0, 18, 43)
    elif kind == "zero":
        a[:, 3:9] = 0.0
    elif kind == "tiny":
        a *= 1e-120
    elif kind == "huge":
        a *= 1e120
    qm, r = (t.cpu().numpy() for t in gb.qr(torch.from_numpy(a).cuda()))
    c = 20 * np.sqrt(211 * 43) * EPS
    assert np.abs(qm.T @ qm - np.eye(43)).max() <= c
    assert np.linalg.norm(qm @ r - a) <= c * np.linalg.norm(a)


def test_qr_keeps_non_finite_visible():
    a = torch.randn(90, 12, dtype=torch.float64, device="cuda")
    a[17, 4] = float("nan")
    q = gb.qr(a)[0]
    assert bool(torch.isnan(q[:, 4:]).all())
    a[17, 4] = float("inf")
    assert not bool(torch.isfinite(gb.qr(a)[0][:, 4]).all())
