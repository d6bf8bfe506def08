"""Outputs that the FP64 digit products leave to the FMA chain: those on rows and
columns with an infinity or a NaN, in each form of the products (column tiles, K ranges
that are summed, the streaming form) and each form of the chain kernel (listed outputs
of short and long chains, whole blocks)."""

import pytest
import torch

import acetn_gb300 as gb

pytestmark = pytest.mark.gpu

INF, NAN = float("inf"), float("nan")


def normal(m, n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(m, n, generator=g, dtype=torch.float64, device="cuda")


def check(a, b):
    """Non-finite outputs as cuBLAS's, finite ones within the rounding of K terms of unit
    size in random order, 8 sqrt(K) u of the largest."""
    c, ref = gb.matmul(a, b), a @ b
    assert gb._abi.device_status() == 0
    assert torch.equal(c.isnan(), ref.isnan())
    inf = ref.isinf()
    assert torch.equal(c.isinf(), inf) and torch.equal(c[inf], ref[inf])
    fine = ref.isfinite()
    bar = 8 * a.shape[1] ** 0.5 * 1.1e-16 * float(ref[fine].abs().max())
    assert float((c[fine] - ref[fine]).abs().max()) < bar


# several tiles a CTA with a long chain behind each bad row; one tile a CTA; K ranges;
# the streaming form with one and two phases and the long operand on either side
SHAPES = [(6000, 2000, 600), (1300, 1250, 40000), (700, 400, 100), (128, 64, 2881),
          (19, 300, 70001), (30000, 24, 30), (36, 9001, 72), (9000, 100, 150)]


@pytest.mark.parametrize("m,n,k", SHAPES)
def test_bad_rows(m, n, k):
    a, b = normal(m, k, 1), normal(k, n, 2)
    rows = torch.arange(5, m, 97, device="cuda")
    a[rows, (7 * rows) % k] = INF
    a[m - 1, k - 1], a[0, 0] = NAN, -INF
    b[3, n // 2], b[k - 1, n - 1], b[0, 1] = -INF, NAN, 0.0
    check(a, b)


@pytest.mark.parametrize("m,n,k", [(700, 400, 100), (128, 64, 2881), (9000, 100, 150), (30000, 24, 30)])
@pytest.mark.parametrize("every", [1, 3])
def test_many_bad_rows(m, n, k, every):
    """As a state that has diverged: whole blocks of outputs by the chain."""
    a, b = normal(m, k, 3), normal(k, n, 4)
    a[::every, k // 2] = NAN
    a[m // 2] = 1.0
    b[:, n // 2] = 0.5
    check(a, b)


def test_added_to():
    """With beta: parts of a contracted index beyond a gigabyte of digits, whose second
    part adds to the first's stored outputs."""
    a, b = normal(20, 4000001, 5), normal(4000001, 24, 6)
    a[3, 17], b[4000000, 5] = INF, -INF
    check(a, b)
