"""FP64 density matrices and norm tensors of a state whose environment legs carry opposite
powers of two on their two sides: an exact change of gauge, so nothing may change beyond
the rounding of sums of positive terms (the contractions have several modes a side, strided
operands and all forms of the digit products)."""

import pytest
import torch

import acetn_gb300 as gb

pytestmark = pytest.mark.gpu


def state(D, chi, gauge):
    g = torch.Generator(device="cuda").manual_seed(D + chi)

    def rnd(*shape):
        return torch.rand(*shape, generator=g, dtype=torch.float64, device="cuda") + 0.1

    st = gb.IpepsState(2, 2, {"phys": 2, "bond": D, "chi": chi})
    A, C, E = rnd(D, D, D, D, 2), [rnd(chi, chi) for _ in range(4)], [rnd(chi, chi, D, D) for _ in range(4)]
    for k in range(4):  # C[k]'s second leg on E[k]'s first, E[k]'s second on C[k + 1]'s first
        e = torch.randint(-gauge, gauge + 1, (chi,), generator=g, device="cuda")
        up, down = (torch.ldexp(torch.ones(chi, dtype=torch.float64, device="cuda"), t) for t in (e, -e))
        C[k], C[(k + 1) % 4] = C[k] * up, C[(k + 1) % 4] * down[:, None]
        E[k] = E[k] * down[:, None, None, None] * up[:, None, None]
    for site in st.site_list:
        st[site] = {"A": A, "C": list(C), "E": list(E)}
    return st


def outputs(st):
    rdm = gb.RDM(st)
    return [rdm[st.site_list[0]], rdm[st.bond_list[0]], rdm[st.bond_list[-1]]]


@pytest.mark.parametrize("D,chi", [(4, 64), (5, 50), (3, 90)])
def test_gauge(D, chi):
    """Every output is a sum of positive products of 15 tensors' entries, over four or five
    contractions of at most chi^2 D^2 terms: 60 sqrt(chi^2 D^2) 2^-53 of itself at most."""
    plain, turned = outputs(state(D, chi, 0)), outputs(state(D, chi, 45))
    assert gb._abi.device_status() == 0
    for a, b in zip(plain, turned):
        rel = float(((a - b).abs() / a.abs()).max())
        assert rel < 60 * chi * D * 2.0 ** -53, rel
