"""FP64 contractions by exact digit products, at the edges of their tiles,
chunks and K ranges, against sums in extended precision.

Bound: with rows scaled to below 1 by the next power of two (at most twice the
largest entry), the dropped products are at most 7 K 2^14 / 2^76 and the
rounding of the operands 2 K 2^-63 of the scales' product, which is at most
4 max|a| max|b|: together below K 2^-57 max|a| max|b|; the result is rounded
once (K ranges that are summed add one rounding each, at most 12)."""

import numpy as np
import pytest
import torch

import acetn_gb300 as gb
from oracle import ctm_oracle as orc

pytestmark = pytest.mark.gpu


def product(a, b):
    """a @ b with about 64 extra bits: exact products of 26-bit halves."""
    def halves(x):
        c = x * (2.0 ** 27 + 1)
        h = c - (c - x)
        return h, x - h
    if np.finfo(np.longdouble).nmant > 100:  # IEEE quadruple
        return a.astype(np.longdouble) @ b.astype(np.longdouble)
    (ah, al), (bh, bl) = halves(a), halves(b)
    return sum((x.astype(np.longdouble) @ y.astype(np.longdouble)) for x in (ah, al) for y in (bh, bl))


def check(a, b, c, splits=12):
    ref = product(a, b)
    k = a.shape[1]
    scale = np.abs(a).max(1)[:, None] * np.abs(b).max(0)[None, :]
    bound = k * 2.0 ** -57 * scale + (1 + splits) * 2.0 ** -53 * np.abs(ref).astype(float)
    err = np.abs((c - ref).astype(float))
    assert np.all(err <= bound), float((err / np.maximum(bound, 1e-300)).max())
    return err


def run(a, b):
    out = gb.matmul(torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()).cpu().numpy()
    assert gb._abi.device_status() == 0
    return out


# rows, columns, contracted: each of at least 2e7 multiply-adds, so that all of
# them take the digit form
SHAPES = [(1300, 1000, 16), (1280, 1024, 17), (1111, 640, 31), (1024, 640, 32), (977, 651, 33),
          (640, 500, 64), (513, 257, 191), (512, 256, 192), (511, 255, 193), (384, 260, 255),
          (385, 259, 256), (129, 700, 257), (128, 640, 384), (127, 65, 2500), (16, 250, 5184),
          (4000, 16, 400), (72, 1500, 200), (1500, 49, 300), (160, 160, 1600), (161, 90, 5000),
          (128, 64, 2881)]


@pytest.mark.parametrize("m,n,k", SHAPES)
def test_edges(m, n, k):
    rng = np.random.default_rng(m + n + k)
    a, b = rng.standard_normal((m, k)), rng.standard_normal((k, n))
    a[m // 2] = 0.0
    b[:, n // 3] *= 1e-200
    check(a, b, run(a, b))


@pytest.mark.parametrize("kind", ["graded", "extreme", "ones", "tiny", "huge", "mixed"])
def test_values(kind):
    rng = np.random.default_rng(5)
    m, n, k = 300, 200, 400
    a, b = rng.standard_normal((m, k)), rng.standard_normal((k, n))
    if kind == "graded":  # over 60 binary orders within each row
        a *= 2.0 ** -rng.integers(0, 60, (m, k))
        b *= 2.0 ** -rng.integers(0, 60, (k, n))
    elif kind == "extreme":  # every lower digit -128: the largest partial sums
        x = -sum(128 * 256.0 ** -i for i in range(1, 8)) * 2.0 ** -6
        a, b = np.full((m, k), x), np.full((k, n), x)
        a[:, 0], b[0] = 0.999, 0.999
    elif kind == "ones":
        a, b = np.full((m, k), 1 - 2.0 ** -53), np.full((k, n), -(1 - 2.0 ** -53))
    elif kind == "tiny":
        a, b = a * 1e-160, b * 1e-140
    elif kind == "huge":
        a, b = a * 1e150, b * 1e150
    elif kind == "mixed":
        a *= 2.0 ** rng.integers(-400, 400, (m, 1))
        b *= 2.0 ** rng.integers(-400, 400, (1, n))
    check(a, b, run(a, b))


def test_closer_than_the_fma_chain():
    rng = np.random.default_rng(6)
    for m, n, k, grade in ((700, 400, 100, 0), (300, 200, 2000, 0), (500, 400, 144, 30)):
        a, b = rng.standard_normal((m, k)), rng.standard_normal((k, n))
        g = 2.0 ** (-grade * np.arange(k) / k)
        a, b = a * g, b * g[:, None]
        err = check(a, b, run(a, b))
        chain = np.zeros((m, n))
        for i in range(k):  # rounded products, so up to twice the FMA chain's error
            chain += a[:, i:i + 1] * b[i:i + 1]
        ref = product(a, b)
        assert np.linalg.norm(err) <= np.linalg.norm((chain - ref).astype(float))


def test_non_finite():
    rng = np.random.default_rng(7)
    a, b = rng.standard_normal((400, 300)), rng.standard_normal((300, 256))
    a[3, 5], a[200, 299], b[7, 11], b[0, 255] = np.inf, np.nan, -np.inf, np.nan
    b[5, 100] = 0.0  # inf * 0
    c, ref = run(a, b), a @ b
    assert np.array_equal(np.isnan(c), np.isnan(ref)) and np.array_equal(np.isinf(c), np.isinf(ref))
    bad = ~np.isfinite(ref)
    assert np.array_equal(c[bad & ~np.isnan(ref)], ref[bad & ~np.isnan(ref)])
    assert np.abs(c[~bad] - ref[~bad]).max() < 1e-11


def test_strided_operands():
    """Every orientation of the loaders through the quarter tensors and RDMs of
    a state with uneven legs, against plain torch."""
    st = gb.random_state(4, 40, seed=3)
    g = torch.Generator(device="cuda").manual_seed(1)
    for s in st.site_list:
        st[s]["C"] = [torch.randn(40, 40, generator=g, dtype=torch.float64, device="cuda") for _ in range(4)]
        st[s]["E"] = [torch.randn(40, 40, 4, 4, generator=g, dtype=torch.float64, device="cuda") for _ in range(4)]
    ein = torch.einsum
    for k in range(4):
        s = st[0, 0]
        a = s["A"].permute([(i + k) % 4 for i in range(4)] + [4])
        t = ein("acuU,ealL->cuUelL", ein("ab,bcuU->acuU", s["C"][k], s["E"][k]), s["E"][(k + 3) % 4])
        q = ein("lurdp,cuelRDp->crRedD", a, ein("cuUelL,LURDp->cuelRDp", t, a)).reshape(640, 640)
        mine = gb.ProjectorCalculator.make_quarter_tensor(s, k)[0]
        # chains of 40, 40, 16 and 32 terms in either order: 1e-13 of the largest
        assert float((mine - q / q.abs().max()).abs().max()) < 1e-13


@pytest.mark.parametrize("D,chi", [(4, 61), (4, 64), (5, 41)])
def test_long_rows_of_several_modes(D, chi):
    """The site density matrix sums over chi D chi D terms whose modes lie apart in one
    operand.  Positive entries: a chain of K terms is within K u of the sum, here
    6e4 1.1e-16, six times over 4e-11; a term lost would be 1 in 6e4."""
    rng = np.random.default_rng(chi)
    st = gb.random_state(D, 4, 1, nx=1, ny=1)
    site = st.site_list[0]
    arrays = {"A": rng.uniform(0.5, 1.5, (D, D, D, D, 2)) / D**2,
              "C": [rng.uniform(0.5, 1.5, (chi, chi)) / chi for _ in range(4)],
              "E": [rng.uniform(0.5, 1.5, (chi, chi, D, D)) / chi for _ in range(4)]}
    st.set_site(site, **arrays)
    mine = gb.RDM(st, "fp64")[site].cpu().numpy()
    assert np.abs(mine / orc.site_rdm(arrays) - 1.0).max() < 4e-11


# long side, small side, contracted: the streaming kernel's groups of columns
# (16, 32, 48, 64 wide), blocks of 16 indices, one and several phases
STREAM = [(80000, 16, 16), (8192, 128, 20), (12001, 72, 36), (17000, 32, 37), (9000, 64, 48),
          (9999, 33, 64), (12800, 17, 96), (8200, 36, 72), (8193, 48, 81), (10000, 49, 49),
          (8192, 96, 33), (8300, 100, 129), (9001, 128, 64), (8192, 65, 176), (8320, 16, 191),
          (12288, 40, 192), (30000, 24, 30)]


@pytest.mark.parametrize("long,short,k", STREAM)
@pytest.mark.parametrize("second", [False, True])
def test_long_operands(long, short, k, second):
    assert long * short * k >= 2e7 and long >= 8192  # the streaming route
    rng = np.random.default_rng(long + short + k)
    a = rng.standard_normal((long, k)) * 2.0 ** rng.integers(-30, 30, (long, 1))
    b = rng.standard_normal((k, short))
    a[7] = 0.0
    rows = np.unique(np.concatenate([np.arange(140), rng.integers(0, long, 200),
                                     np.arange(long - 140, long)]))
    c = run(np.ascontiguousarray(b.T), np.ascontiguousarray(a.T)).T if second else run(a, b)
    check(a[rows], b, c[rows], splits=0)
    scale = np.abs(a).max(1)[:, None] * np.abs(b).max(0)[None, :]  # and every entry loosely
    assert np.all(np.abs(c - a @ b) <= k * 2.0 ** -50 * scale)


def test_long_operand_non_finite_and_extreme():
    rng = np.random.default_rng(9)
    a, b = rng.standard_normal((9000, 50)), rng.standard_normal((50, 60))
    a[5, 3], a[8999, 49], b[7, 59] = np.inf, np.nan, -np.inf
    b[3, 10] = 0.0
    c, ref = run(a, b), a @ b
    assert np.array_equal(np.isnan(c), np.isnan(ref)) and np.array_equal(np.isinf(c), np.isinf(ref))
    fine = np.isfinite(ref)
    assert np.abs(c[fine] - ref[fine]).max() < 1e-12
    x = -sum(128 * 256.0 ** -i for i in range(1, 8)) * 2.0 ** -6
    for k in (36, 192):
        a, b = np.full((8192, k), x), np.full((k, 80), x)
        a[:, 0], b[0] = 0.999, 0.999
        check(a[:200], b, run(a, b)[:200], splits=0)
