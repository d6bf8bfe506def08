"""The FP64 reciprocal and square root from FP32 seeds, against extended precision, at both
ends of the binade, odd and even exponents and the limits of the fallback.

Bounds (derived beside the code): the reciprocal and the root within one ulp; beta, the
reciprocal of d - alpha a with that difference rounded once, within 2^-51.4 of it."""

import ctypes

import numpy as np
import pytest
import torch

from acetn_gb300 import _abi

pytestmark = pytest.mark.gpu


def seeded(x, y):
    fn = _abi.load().ctm_test_seeded
    fn.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int64, ctypes.c_void_p, ctypes.c_void_p]
    fn.restype = ctypes.c_int
    dx, dy = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
    out = torch.empty(3, len(x), dtype=torch.float64, device="cuda")
    assert fn(dx.data_ptr(), dy.data_ptr(), len(x), out.data_ptr(),
              ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    return out.cpu().numpy()


def mantissas(rng):
    eps = 2.0 ** -52
    ends = [1 + k * eps for k in range(40)] + [2 - k * eps for k in range(1, 40)]
    # around multiples of 2^-23, where the seed's argument jumps
    cuts = [1 + k * 2.0 ** -23 + j * eps for k in (1, 2, 3, 1 << 22, (1 << 23) - 1)
            for j in range(-3, 4)]
    return np.array(ends + cuts + list(rng.uniform(1, 2, 4000)))


@pytest.mark.parametrize("exponent", [-1022, -1021, -1001, -1000, -999, -501, -500, -2, -1, 0, 1, 2,
                                      500, 501, 999, 1000, 1001, 1020, 1021])
def test_against_extended(exponent):
    rng = np.random.default_rng(exponent + 2000)
    x = np.ldexp(mantissas(rng), exponent)
    x = x[x >= 2.0 ** -1022]
    root = np.sqrt(x.astype(np.longdouble))
    y = np.asarray(root * rng.uniform(-1, 1, len(x)), dtype=np.float64)
    y[::7] = 0.0
    y[1::7] = np.asarray(root, dtype=np.float64)[1::7] * (1 - 2.0 ** -52)
    y[2::7] = -y[2::7]
    rec, alpha, beta = seeded(x, y)
    want = 1 / x.astype(np.longdouble)
    ulp = np.spacing(np.abs(want).astype(np.float64)).astype(np.longdouble)
    assert np.all(np.abs(rec - want) <= ulp)
    ulp = np.spacing(root.astype(np.float64)).astype(np.longdouble)
    assert np.all(np.abs(np.abs(alpha) - root) <= ulp)
    assert np.all((alpha < 0) == (y >= 0))
    v = x.astype(np.longdouble) - alpha.astype(np.longdouble) * y.astype(np.longdouble)
    if np.finfo(np.longdouble).nmant < 60:
        pytest.skip("no extended precision")
    fine = np.abs(1 / v) > 2.0 ** -1021
    rel = np.abs(beta[fine] * v[fine] - 1)
    assert np.all(rel <= 2.0 ** -51.4), float(rel.max())


def test_special():
    x = np.array([0.0, np.inf, np.nan, 5e-324])
    _, alpha, beta = seeded(x, np.zeros(4))
    assert alpha[0] == 0 and beta[0] == 0 and np.isnan(alpha[1:3]).all() and np.isnan(beta[1:3]).all()
    assert alpha[3] == 0 and beta[3] == 0
