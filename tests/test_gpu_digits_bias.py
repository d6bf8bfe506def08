"""The rounding of the FP64 streaming product's fixed-point sums."""

import numpy as np
import pytest
import torch

import acetn_gb300 as gb
from test_gpu_digits import product

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k", [(60, 36), (60, 80), (40, 150)])
def test_no_bias(n, k):
    """The streaming form keeps 57, 56 or 55 bits below the scales: to nearest, so the
    mean error over 16000 outputs and more is far below half a unit (one-sided truncation:
    2^-58, 2^-57, 2^-56 of the scales; the final rounding's mean has a deviation below
    2^-62)."""
    rng = np.random.default_rng(k)
    a, b = rng.uniform(-1, 1, (12000, k)), rng.uniform(-1, 1, (k, n))
    a[:, 0], b[0] = 0.9375, 0.9375  # scales of 1
    rows = np.arange(0, 12000, 30)
    c = gb.matmul(torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()).cpu().numpy()
    err = (c[rows] - product(a[rows], b)).astype(float)
    assert abs(err.mean()) < 2.0**-59
