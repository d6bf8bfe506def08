"""Workspace of the FP64 SVD of a long matrix: no copies of it for the Householder fallback
that its Cholesky-QR does not use (the size query needs no GPU)."""

import ctypes
import os

import pytest

import acetn_gb300 as gb


@pytest.mark.skipif(not os.path.exists(os.path.join(os.path.dirname(gb.__file__), "lib")),
                    reason="library not built")
@pytest.mark.parametrize("rows,cols", [(4000, 160), (160, 4000)])
def test_long_matrix(rows, cols):
    """Three copies (the input as rows, Q and the next stage's), the digits of both operands
    of its Gram matrix (two each, a ninth of that in masks and scales), the partial sums of
    the latter (half a copy) and small matrices (14 of 160 x 160): nine, not eleven."""
    fn = gb._abi.load().ctm_svd_f64
    size = ctypes.c_size_t(0)
    assert fn(None, ctypes.c_int64(rows), ctypes.c_int64(cols), None, None, None, None,
              ctypes.byref(size), None) == 0
    assert size.value < 9.5 * 8 * rows * cols
