"""``svd_f32`` beyond q = 256, where the Jacobi rows are spread over a cluster (257: an
odd number in registers; 288: the last of that width; 289 and 400: rows re-read; 700:
beyond the cluster's shared memory), held to the bars of the smaller sizes: singular
values to 2e-6 of s0, U orthogonal to 5e-6, the reconstruction to 1e-5."""

import numpy as np
import pytest
import torch

import acetn_gb300 as gb
from acetn_gb300 import _abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,q", [(1200, 257), (1300, 288), (1300, 289), (1600, 400), (1500, 700)])
def test_svd_f32_spread(n, q):
    rng = np.random.default_rng(q)
    v, _ = np.linalg.qr(rng.standard_normal((n, q)))
    u, _ = np.linalg.qr(rng.standard_normal((q, q)))
    s_true = np.geomspace(1.0, 2e-4, q)
    bt = torch.from_numpy((v * s_true) @ u.T).to("cuda", torch.float32)
    _abi.device_status()
    U, S, V = gb.linalg.svd_f32(bt)
    torch.cuda.synchronize()
    assert _abi.device_status() == 0
    b32 = bt.double().cpu().numpy().T
    s_ref = np.linalg.svd(b32, compute_uv=False)
    U, S, V = U.cpu().numpy(), S.cpu().numpy(), V.double().cpu().numpy()
    assert np.abs(S - s_ref).max() / s_ref[0] < 2e-6
    assert np.abs(U.T @ U - np.eye(q)).max() < 5e-6
    assert np.abs((U * S) @ V.T - b32).max() / np.abs(b32).max() < 1e-5
