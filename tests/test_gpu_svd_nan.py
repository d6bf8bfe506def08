"""FP64 SVD of a state that has diverged: no output keeps what its buffer held before."""

import pytest
import torch

import acetn_gb300 as gb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n", [(22, 80), (40, 40), (60, 30), (144, 144), (1500, 90)])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_every_output_is_written(m, n, bad):
    g = torch.Generator(device="cuda").manual_seed(m)
    a = torch.randn(m, n, generator=g, dtype=torch.float64, device="cuda")
    a[m // 2, n // 3] = bad
    a[m - 1, n // 2] = bad
    r, mark = min(m, n), 7.25
    out = [torch.full(s, mark, dtype=torch.float64, device="cuda") for s in ((m, r), (r,), (n, r))]
    gb._abi.call("ctm_svd_f64", [gb._abi.ptr(a), m, n] + [gb._abi.ptr(t) for t in out], a.device)
    gb._abi.device_status()  # (reads and clears the flags)
    assert not any(bool((t == mark).any()) for t in out)
    assert not bool(out[1].isfinite().all())
