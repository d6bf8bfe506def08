"""FP64 SVD of long matrices that the Cholesky route gives up (values down to 1e-15): again in
one cluster where the rows fit, else in global memory; the bounds of the SVD tests."""

import numpy as np
import pytest
import torch

import acetn_gb300 as gb
from test_gpu_svd_f64 import check, matrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n", [(60, 1200), (601, 100), (160, 1100), (700, 100), (66, 4000)])
@pytest.mark.parametrize("kind", ["steep", "deficient"])
def test_given_up(m, n, kind):
    rng = np.random.default_rng(m)
    r = min(m, n)
    if kind == "steep":
        u, v = np.linalg.qr(rng.standard_normal((m, r)))[0], np.linalg.qr(rng.standard_normal((n, r)))[0]
        a = np.ascontiguousarray((u * 10.0 ** (-15 * np.arange(r) / (r - 1))) @ v.T)
    else:
        a = np.ascontiguousarray(matrix(m, r // 3, "random") @ matrix(r // 3, n, "random"))
    u, s, v = (t.cpu().numpy() for t in gb.svd(torch.from_numpy(a).cuda()))
    assert gb._abi.device_status() == 0
    c = check(a, u, s, v)
    short = u if m <= n else v
    assert np.abs(short.T @ short - np.eye(r)).max() <= c
