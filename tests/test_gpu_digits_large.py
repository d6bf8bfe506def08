"""FP64 contractions whose digits would exceed a gigabyte are done in parts: halves of
the rows, of the columns and of the contracted index (one mode, and the several modes
of a site density matrix).  Rounding: a chain of K terms of unit size is within K u, in
random order sqrt(K) u, of the exact sum; the bars are 8 times the latter relative to
the largest entry (K = 4e6: 2e3 * 1.1e-16 * 8 = 2e-12)."""

import numpy as np
import pytest
import torch

import acetn_gb300 as gb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(70001, 17, 1001), (19, 66000, 1003), (20, 24, 4000001)])
def test_parts(m, n, k):
    g = torch.Generator(device="cuda").manual_seed(m)
    a = torch.randn(m, k, generator=g, dtype=torch.float64, device="cuda")
    b = torch.randn(k, n, generator=g, dtype=torch.float64, device="cuda")
    ref = a @ b
    diff = (gb.matmul(a, b) - ref).abs().max() / ref.abs().max()
    assert float(diff) < 8 * k**0.5 * 1.1e-16


def test_parts_of_several_modes():
    D, chi = 6, 180
    g = torch.Generator(device="cuda").manual_seed(1)

    def positive(*shape):
        return (torch.rand(*shape, generator=g, dtype=torch.float64, device="cuda") + 0.5) / shape[0]

    st = gb.random_state(D, 4, 1, nx=1, ny=1, device="cuda")
    s = st.site_list[0]
    A, C = positive(D, D, D, D, 2), [positive(chi, chi) for _ in range(4)]
    E = [positive(chi, chi, D, D) for _ in range(4)]
    st[s] = {"A": A, "C": C, "E": E}
    mine = gb.RDM(st, "fp64")[s]
    ein = torch.einsum
    left = ein("aclL,eadD->clLedD", ein("ab,bclL->aclL", C[3], E[3]), E[2])
    left = ein("clLedD,LURDP->cledURP", left, A)
    right = ein("ec,bcrR->ebrR", C[1], ein("ab,carR->bcrR", C[2], E[1]))
    right = ein("ebrR,aeuU->brRauU", right, ein("ab,bcuU->acuU", C[0], E[0]))
    ref = ein("ruldP,lurdp->Pp", ein("erRcuU,cledURP->ruldP", right, left), A)
    # positive entries: at most K u relative, K = 36 * 180^2
    assert float((mine / ref - 1).abs().max()) < 36 * 180**2 * 1.1e-16
