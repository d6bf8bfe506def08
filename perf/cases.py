"""Workloads of the framework, from the smallest environment to the largest.

Every case goes through the public entry points (``ctmrg``,
``DirectionalMover``, ``BatchedCTMRG``, ``RDM``, ``build_norm_tensor``,
``ALSSolver``, the randomized SVDs) on environments that a plain torch CTMRG
below has grown from seeded random site tensors, so that spectra and entry
sizes are those of a run in progress.

Singular vectors carry free signs, and the environment's legs carry them on,
so the cases that renormalize return the reduced density matrices (what a
program measures next; signs cancel), and the SVDs fix each singular pair's
sign as a program does that compares vectors.  With a randomized SVD the
signs of one move's legs decide which test matrix a later move in the other
direction sees, so whole iterations run with the exact SVD and the cases with
a randomized one renormalize along one axis.
"""

import importlib
import math

import torch

gb = importlib.import_module("ace-tn_gb300")
ein = torch.einsum


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # the tutorial-sized Heisenberg run: the column half of an iteration
        # and a measurement; the cost is the number and the latency of small
        # launches
        dict(name="columns_d2_chi20", kind="columns", D=2, chi=20, d=2, nx=2, ny=2, bias=0.0,
             projectors="half-system", svd="rsvd", over=2, niter=2),
        # one iteration with full-system projectors and an exact SVD, as used
        # to converge small ground states
        dict(name="iterate_d3_chi16_full", kind="iterate", D=3, chi=16, d=2, nx=2, ny=2, bias=0.0,
             projectors="full-system", svd="full-rank", over=0, niter=0),
        # a transverse-field Ising production run (state near a product state)
        dict(name="columns_d4_chi64", kind="columns", D=4, chi=64, d=2, nx=2, ny=2, bias=0.1,
             projectors="half-system", svd="rsvd", over=2, niter=2),
        # a parameter sweep: several uneven states advanced by one CUDA graph
        dict(name="sweep_4", kind="sweep", D=3, chi=16, D2=2, chi2=30, count=4, d=2),
        # one move at sizes that divide nothing, full-system projectors
        dict(name="move_d5_chi77_full", kind="move", D=5, chi=77, d=2, nx=2, ny=2, k=1,
             precision="fp64", projectors="full-system", over=3, niter=2),
        # the benchmark's own workload in the default precision, one move
        dict(name="move_d6_chi144", kind="move", D=6, chi=144, d=2, nx=2, ny=2, k=0,
             precision="fp64", projectors="half-system", over=16, niter=2),
        # the same in mixed precision, a left/right pair as ctmrg runs it
        dict(name="pair_d6_chi144_mixed", kind="pair", D=6, chi=144, d=2, nx=2, ny=2, k=0,
             precision="mixed", projectors="half-system", over=16, niter=2),
        # the largest environment of the benchmark, mixed precision
        dict(name="move_d8_chi256_mixed", kind="move", D=8, chi=256, d=2, nx=2, ny=2, k=3,
             precision="mixed", projectors="half-system", over=16, niter=2),
        # a measurement on its own: one bond and one site of the large state
        dict(name="rdm_d6_chi144", kind="rdm", D=6, chi=144, d=2, k=2, precision="fp64"),
        # the full update's environment of one bond
        dict(name="norm_d4_chi64", kind="norm", D=4, chi=64, d=2, nD=8, k=1),
        # the full update's least-squares loop for a D=6 bond
        dict(name="als_d6", kind="als", nD=12, bD=6, pD=2, iters=10),
        # a randomized SVD of a product of two tall factors, odd sizes
        dict(name="svd_1100x1323", kind="svd", factors=2, m=1100, k=1211, n=1323, q=90, niter=2),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["columns", "columns", "iterate", "move", "move", "mixed", "rdm", "rdm",
                       "norm", "als", "svd", "svd", "sweep"])
    d = rng.choice([2, 2, 2, 3])
    if kind in ("columns", "iterate"):
        D = rng.choice([2, 3, 4])
        nx, ny = rng.choice([(2, 2), (2, 2), (2, 3), (3, 2)])
        shape = dict(kind=kind, D=D, d=d, nx=nx, ny=ny, bias=rng.choice([0.0, 0.1, 0.3]))
        if kind == "iterate":
            return dict(shape, chi=_log(rng, 8, {2: 44, 3: 20, 4: 12}[D]), svd="full-rank",
                        over=0, niter=0, projectors=rng.choice(["half-system", "full-system"]))
        return dict(shape, projectors="half-system", chi=_log(rng, 8, {2: 60, 3: 72, 4: 60}[D]), svd="rsvd",
                    over=rng.choice([0, 2, 5, 16]), niter=rng.choice([1, 2]))
    if kind == "move":
        D = rng.choice([4, 5, 6])
        full = D < 6 and rng.random() < 0.3
        return dict(kind="move", D=D, chi=_log(rng, 40, 100 if full else 144), d=2, nx=2, ny=2,
                    k=rng.randrange(4), precision="fp64",
                    projectors="full-system" if full else "half-system",
                    over=rng.choice([2, 7, 16]), niter=2)
    if kind == "mixed":
        D = rng.choice([3, 4, 5, 6, 7])
        return dict(kind=rng.choice(["move", "pair"]), D=D, chi=_log(rng, 48, 200), d=2, nx=2,
                    ny=2, k=rng.randrange(2), precision="mixed", projectors="half-system",
                    over=rng.choice([2, 16]), niter=2)
    if kind == "rdm":
        D = rng.choice([2, 3, 4, 5, 6])
        return dict(kind="rdm", D=D, chi=_log(rng, 16, 144), d=2 if D > 4 else d,
                    k=rng.randrange(4), precision="fp64")
    if kind == "norm":
        D = rng.choice([2, 3, 4, 5])
        return dict(kind="norm", D=D, chi=_log(rng, 16, 90), d=d, nD=D * d - rng.randrange(2),
                    k=rng.randrange(4))
    if kind == "als":
        bD, pD = rng.choice([2, 3, 4, 5, 6]), rng.choice([2, 3])
        return dict(kind="als", nD=bD * pD, bD=bD, pD=pD, iters=rng.choice([4, 7, 10]))
    if kind == "svd":
        m, k, n = (_log(rng, 60, 2600) for _ in range(3))
        return dict(kind="svd", factors=rng.choice([1, 2, 2, 4]), m=m, k=k, n=n,
                    q=min(m, k, n, _log(rng, 8, 160)), niter=rng.choice([0, 1, 2]))
    return dict(kind="sweep", D=3, chi=_log(rng, 9, 20), D2=2, chi2=_log(rng, 12, 40),
                count=rng.choice([3, 4, 5]), d=2)


# ---------------------------------------------------------------- CTMRG in plain torch
# Legs and index order as the framework's states have them: A (l, u, r, d, p),
# C[k] (chi, chi), E[k] (chi, chi, D, D); direction k turns A by k legs.
def _turn(A, k):
    return A.permute([(i + k) % 4 for i in range(4)] + [4])


def _quarter(s, k):
    a, c, e1, e2 = _turn(s["A"], k), s["C"][k % 4], s["E"][(k + 3) % 4], s["E"][k % 4]
    t = ein("acuU,ealL->cuUelL", ein("ab,bcuU->acuU", c, e2), e1)
    q = ein("lurdp,cuelRDp->crRedD", a, ein("cuUelL,LURDp->cuelRDp", t, a))
    q = q.reshape(q.shape[0] * q.shape[1] ** 2, -1)
    return q / q.abs().max()


def _chain(fs, x):
    for f in reversed(fs):
        x = f @ x
    return x


def _rsvd(fs, q, niter, omega):
    ft = [f.T for f in reversed(fs)]
    y = _chain(fs, omega)
    for _ in range(niter):
        z = _chain(ft, torch.linalg.qr(y)[0])
        if len(fs) == 4:
            z = torch.linalg.qr(z)[0]
        y = _chain(fs, z)
    qm = torch.linalg.qr(y)[0]
    b = qm.T
    for f in fs:
        b = b @ f
    u, s, vh = torch.linalg.svd(b, full_matrices=False)
    return qm @ u, s, vh.T


def _projectors(st, sites, k, chi, cfg, omega):
    """(P1, P2) of one row, each (chi', D, D, chi)."""
    D = st[sites[0]]["A"].shape[0]
    full = cfg["projectors"] == "full-system"
    q1, q4 = _quarter(st[sites[0]], k), _quarter(st[sites[3]], k + 3)
    left, right = [q1], [q4]
    if full:
        left = [_quarter(st[sites[1]], k + 1), q1]
        right = [q4, _quarter(st[sites[2]], k + 2)]
    if cfg["svd"] == "rsvd":
        fs = left + right
        q = min(chi + cfg["over"], fs[0].shape[0], fs[-1].shape[1])
        u, s, v = _rsvd(fs, q, cfg["niter"], omega(fs[-1].shape[1], q))
    else:
        if full:
            left, right = [left[0] @ left[1]], [right[0] @ right[1]]
            left, right = [left[0] / left[0].abs().max()], [right[0] / right[0].abs().max()]
        f = left[0] @ right[0]
        u, s, vh = torch.linalg.svd(f / f.abs().max(), full_matrices=False)
        v = vh.T
    s = s / s[0]
    n = min(chi, int((s > cfg.get("cutoff", 1e-12)).sum()))
    w = s[:n].rsqrt()
    p1, p2 = _chain([f.T for f in reversed(left)], u[:, :n] * w), _chain(right, v[:, :n] * w)
    return p1.reshape(-1, D, D, n), p2.reshape(-1, D, D, n)


def _unit(x):
    return x / x.norm()


def _renormalize(s, k, p1i, p2j, p2i, p1j):
    """The corner, corner and edge that replace C[k+3], C[k], E[k+3]."""
    t = ein("ablL,bc->alLc", s["E"][(2 + k) % 4], s["C"][(3 + k) % 4])
    c1 = ein("alLc,clLx->ax", t, p1i)
    c2 = ein("arRx,acrR->xc", p2j, ein("ab,bcrR->acrR", s["C"][k % 4], s["E"][k % 4]))
    a = _turn(s["A"], k)
    t = ein("LURDP,alLuUx->RDPalux", a, ein("ablL,buUx->alLuUx", s["E"][(3 + k) % 4], p1j))
    e = ein("rdRDax,adDy->yxrR", ein("lurdp,RDpalux->rdRDax", a, t), p2i)
    return _unit(c1), _unit(c2), _unit(e)


def _rows(k, idx, nx, ny):
    """For each row of move k: the four sites of its projector pair, the site
    read, the site written, and the rows of its two projector pairs."""
    out = []
    for r in range(ny if k % 2 == 0 else nx):
        x, y = (idx, r) if k % 2 == 0 else (r, idx)
        dx, dy = ((1, -1), (-1, -1), (-1, 1), (1, 1))[k]
        x2, y2 = (x + dx) % nx, (y + dy) % ny
        if k % 2 == 0:
            out.append(([(x, y), (x2, y), (x2, y2), (x, y2)], (x, y), (x2, y), r,
                        (r + (1 if k == 0 else -1)) % ny))
        else:
            out.append(([(x, y), (x, y2), (x2, y2), (x2, y)], (x, y), (x, y2), r,
                        (r + (1 if k == 1 else -1)) % nx))
    return out


def _move(st, k, idx, nx, ny, chi, cfg, omega):
    rows = _rows(k, idx, nx, ny)
    pr = [_projectors(st, sites, k, chi, cfg, omega) for sites, *_ in rows]
    new = [_renormalize(st[s1], k, pr[i][0], pr[j][1], pr[i][1], pr[j][0])
           for _, s1, _, i, j in rows]
    for (_, _, s2, _, _), (c1, c2, e) in zip(rows, new):
        st[s2]["C"][(3 + k) % 4], st[s2]["C"][k], st[s2]["E"][(3 + k) % 4] = c1, c2, e


def _sweep(nx, ny):
    return ([m for x in range(nx) for m in ((0, x), (2, (nx - x + 1) % nx))]
            + [m for y in range(ny) for m in ((1, (ny - y + 1) % ny), (3, y))])


def _site_rdm(s):
    (c1, c2, c3, c4), (e1, e2, e3, e4), a = s["C"], s["E"], s["A"]
    t1 = ein("aclL,eadD->clLedD", ein("ab,bclL->aclL", c4, e4), e3)
    t1 = ein("clLedD,LURDP->cledURP", t1, a)
    t3 = ein("ec,bcrR->ebrR", c2, ein("ab,carR->bcrR", c3, e2))
    t3 = ein("ebrR,aeuU->brRauU", t3, ein("ab,bcuU->acuU", c1, e1))
    return ein("ruldP,lurdp->Pp", ein("erRcuU,cledURP->ruldP", t3, t1), a)


def _bond_halves(s1, s2, k):
    """The two open halves of a bond before the site tensors close them."""
    C1, E1, C2, E2 = s1["C"], s1["E"], s2["C"], s2["E"]
    k0, k1, k2, k3 = (j % 4 for j in range(k, k + 4))
    r = ein("acrR,eauU->crReuU", ein("ab,bcrR->acrR", C1[k1], E1[k1]), E1[k0])
    l = ein("acuU,ealL->cuUelL", ein("ab,bcuU->acuU", C2[k0], E2[k0]), E2[k3])
    ra = ein("ab,bfdD->afdD", C1[k2], E1[k2])
    la = ein("ae,fadD->efdD", C2[k3], E2[k2])
    return r, l, ra, la


def _bond_rdm(s1, s2, k):
    r, l, ra, la = _bond_halves(s1, s2, k)
    a1, a2 = _turn(s1["A"], k), _turn(s2["A"], k)
    r = ein("creuLDP,lurdp->ceLDPldp", ein("crReuU,LURDP->creuLDP", r, a1), a1)
    r = ein("afdD,acLDPldp->fcLPlp", ra, r)
    l = ein("cuelRDQ,lurdq->ceRDQrdq", ein("cuUelL,LURDQ->cuelRDQ", l, a2), a2)
    l = ein("efdD,ceRDQrdq->fcRQrq", la, l)
    return ein("fcRPrp,fcRQrq->PQpq", r, l)


def _norm_tensor(s1, s2, k, q1, q2):
    r, l, ra, la = _bond_halves(s1, s2, k)
    r = ein("creuDY,rduy->ceDYdy", ein("crReuU,RDUY->creuDY", r, q1), q1)
    r = ein("afdD,aeDYdy->feYy", ra, r)
    l = ein("cuelXD,dlux->ceXDxd", ein("cuUelL,DLUX->cuelXD", l, q2), q2)
    l = ein("bfdD,cbXDxd->fcXx", la, l)
    return ein("fcYy,fcXx->yxYX", r, l)


# ---------------------------------------------------------------- inputs
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, dtype=torch.float64, device="cuda")


def _environment(D, chi, d, nx, ny, bias, seed):
    """Seeded site tensors of unit norm and their environment after the
    iterations that bring it to chi and one more where that is cheap.  Grown
    in float32 (an environment in mid-run, not a converged one, is wanted);
    the last bits are filled with noise, as float64 entries have them."""
    g = _generator(seed)
    st = {}
    for x in range(nx):
        for y in range(ny):
            A = _randn(g, D, D, D, D, d)
            A[0, 0, 0, 0, 0] += bias * A.numel() ** 0.5
            A = A / A.norm()
            a = A.float()
            C, E = [], []
            for k in range(4):
                ak = _turn(a, k)
                C.append(_unit(ein("lurdp,luRDp->dDrR", ak, ak).reshape(D * D, D * D)))
                E.append(_unit(ein("lurdp,LuRDp->lLrRdD", ak, ak).reshape(D * D, D * D, D, D)))
            st[x, y] = {"A": a, "C": C, "E": E, "A64": A}
    cfg = dict(projectors="half-system", svd="rsvd", over=4, niter=1, cutoff=1e-9)

    def omega(n, q):
        return _randn(g, n, q).float()

    width = D * D
    while True:
        for k, idx in _sweep(nx, ny):
            _move(st, k, idx, nx, ny, chi, cfg, omega)
        width = min(chi, width * D * D)
        if width >= chi:
            break
    if D < 5:
        for k, idx in _sweep(nx, ny):
            _move(st, k, idx, nx, ny, chi, cfg, omega)

    def fill(t):
        t = t.double()
        return (t * (1 + 2.0 ** -26 * _randn(g, *t.shape))).contiguous()

    return {s: {"A": v["A64"].contiguous(), "C": [fill(t) for t in v["C"]],
                "E": [fill(t) for t in v["E"]]} for s, v in st.items()}


def _state(sites, nx, ny, D, chi, d):
    """A state over the given tensors (moves replace list entries, never
    write into the tensors)."""
    st = gb.IpepsState(nx, ny, {"phys": d, "bond": D, "chi": chi})
    for s, v in sites.items():
        st[s] = {"A": v["A"], "C": list(v["C"]), "E": list(v["E"])}
    return st


def _config(case):
    return gb.CTMRGConfig(steps=1, projectors=case.get("projectors", "half-system"),
                          svd_type=case.get("svd", "rsvd"), rsvd_niter=case.get("niter", 2),
                          rsvd_oversampling=case.get("over", 2), disable_progressbar=True,
                          precision=case.get("precision", "fp64"))


def _sweep_sizes(case):
    return [(case["D"], case["chi"]) if i % 2 == 0 else (case["D2"], case["chi2"] - i)
            for i in range(case["count"])]


def _matrices(case, seed):
    """Factors whose product has a spectrum falling by a fixed ratio per
    index, as enlarged corners have it."""
    g = _generator(seed)
    m, k, n = case["m"], case["k"], case["n"]
    r = min(m, k, n)
    s = 10.0 ** (-6.0 * torch.arange(r, device="cuda", dtype=torch.float64) / r)
    u = torch.linalg.qr(_randn(g, m, r))[0]
    v = torch.linalg.qr(_randn(g, n, r))[0]
    if case["factors"] == 1:
        return [((u * s) @ v.T).contiguous()]
    w = torch.linalg.qr(_randn(g, k, r))[0]
    h = s.sqrt()
    two = [((u * h) @ w.T).contiguous(), ((w * h) @ v.T).contiguous()]
    if case["factors"] == 2:
        return two
    turn = torch.linalg.qr(_randn(g, k, k))[0]
    return [two[0], turn.contiguous(), turn.T.contiguous(), two[1]]


def _als_inputs(case, seed):
    nD, bD, pD = case["nD"], case["bD"], case["pD"]
    g = _generator(seed)
    n = _randn(g, nD * nD, 2 * nD * nD) / nD
    n12 = (n @ n.T + 0.1 * torch.eye(nD * nD, device="cuda", dtype=torch.float64))
    a1, a2 = _randn(g, nD, bD, pD), _randn(g, nD, bD, pD)
    s = 10.0 ** (-1.5 * torch.arange(bD, device="cuda", dtype=torch.float64) / bD)
    a12 = ein("yup,xuq->yxpq", a1 * s[:, None], a2)
    gate = torch.eye(pD * pD, device="cuda", dtype=torch.float64) + 0.2 * _randn(g, pD * pD, pD * pD)
    a12g = ein("yxpq,pqrs->yxrs", a12, gate.reshape(pD, pD, pD, pD))
    return n12.reshape(nD, nD, nD, nD).contiguous(), a12g.contiguous()


class _ALSConfig:
    als_tol, als_method, als_epsilon = 0.0, "cholesky", 1e-12

    def __init__(self, iters):
        self.als_niter = iters


def prepare(case, seed):
    kind = case["kind"]
    torch.manual_seed(seed)
    st = {"case": case, "seed": int(seed)}
    if kind == "svd":
        return {**st, "mats": _matrices(case, seed)}
    if kind == "als":
        return {**st, "inputs": _als_inputs(case, seed)}
    if kind == "sweep":
        states = []
        for i, (D, chi) in enumerate(_sweep_sizes(case)):
            env = _environment(D, chi, case["d"], 2, 2, 0.3, 100 * seed + i)
            states.append(_state(env, 2, 2, D, chi, case["d"]))
        cfg = _config(dict(svd="full-rank"))
        return {**st, "batch": gb.BatchedCTMRG(states, cfg).capture(warmup=1)}
    nx, ny = case.get("nx", 2), case.get("ny", 2)
    st["sites"] = _environment(case["D"], case["chi"], case["d"], nx, ny, case.get("bias", 0.0),
                               seed)
    if kind == "norm":
        g = _generator(seed + 7)
        D, nD = case["D"], case["nD"]
        st["q"] = [torch.linalg.qr(_randn(g, D ** 3, nD))[0].reshape(D, D, D, nD).contiguous()
                   for _ in range(2)]
    if kind in ("iterate", "columns", "move", "pair"):
        st["config"] = _config(case)
        st["mover"] = gb.DirectionalMover(st["config"])
    return st


# ---------------------------------------------------------------- one pass
def _written(case):
    nx, ny, k = case["nx"], case["ny"], case["k"]
    ks = [(k, 0)] if case["kind"] == "move" else [(k, 0), (k + 2, 1)]
    return ks, sorted({row[2] for kk, i in ks for row in _rows(kk, i, nx, ny)})


def _sign(u, s, v):
    top = u.gather(0, u.abs().argmax(0, keepdim=True)).sign()
    return {"U": u * top, "S": s, "V": v * top}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "svd":
        # a program that wants the same test matrix again seeds the generator
        torch.manual_seed(state["seed"])
        f = {1: gb.svd_lowrank, 2: gb.fused_matmul_svd_lowrank,
             4: gb.fused_3matmul_svd_lowrank}[case["factors"]]
        return _sign(*f(*state["mats"], q=case["q"], niter=case["niter"]))
    if kind == "als":
        n12, a12g = state["inputs"]
        a1, a2 = gb.ALSSolver(n12, a12g, (case["nD"], case["bD"], case["pD"]),
                              _ALSConfig(case["iters"])).solve()
        return ein("yup,xuq->yxpq", a1, a2)  # the bond index has a free gauge
    if kind == "sweep":
        state["batch"].replay(1)
        return [gb.RDM(st)[0, 0] for st in state["batch"].states]
    nx, ny = case.get("nx", 2), case.get("ny", 2)
    st = _state(state["sites"], nx, ny, case["D"], case["chi"], case["d"])
    if kind == "rdm":
        rdm = gb.RDM(st, case["precision"])
        return {"bond": rdm[gb.Bond(*_bond(case["k"]))], "site": rdm[0, 1]}
    if kind == "norm":
        return gb.build_norm_tensor(st, gb.Bond(*_bond(case["k"])), *state["q"])
    torch.manual_seed(state["seed"])
    if kind in ("iterate", "columns"):
        if kind == "iterate":
            gb.ctmrg(st, state["config"])
        else:
            for x in range(nx):
                state["mover"].left_right_move(st, x, (nx - x + 1) % nx)
        rdm = gb.RDM(st)
        return {"site": [rdm[s] for s in st.site_list], "bond": [rdm[b] for b in st.bond_list]}
    moves, sites = _written(case)
    if kind == "move":
        state["mover"].move(st, *moves[0])
    else:
        state["mover"].move_pair(st, case["k"], moves[0][1], moves[1][1])
    rdm = gb.RDM(st, case["precision"])
    return [rdm[s] for s in sites]


def _bond(k):
    return (0, 0), ((1, 0), (0, 1), (1, 0), (0, 1))[k], k


# ---------------------------------------------------------------- what a pass cannot do without
def _work_move(D, chi, d, rows, q, niter, factors, full_rank):
    n = chi * D * D
    quarter = 2 * chi**3 * D**2 + 2 * chi**3 * D**4 + 4 * chi**2 * D**6 * d
    renorm = 4 * chi**3 * D**4 + 4 * chi**2 * D**6 * d + 8 * chi**3 * D**2
    if full_rank:
        svd = 2.0 * n**3 * (1 if factors == 2 else 3) + 4.0 * n**3
    else:
        svd = 2.0 * n * n * q * factors * (2 + 2 * niter)
    return rows * (factors * quarter + svd + factors * 2.0 * n * n * chi + renorm)


def _work_rdm(D, chi, d, sites, bonds):
    site = 4 * chi**3 * D**4 + 2 * chi**2 * D**6 * d + 2 * chi**2 * D**6 * d
    bond = 2 * (2 * chi**3 * D**4 + 2 * chi**2 * D**6 * d + 2 * chi**2 * D**6 * d * d
                + 2 * chi**3 * D**4 * d * d)
    return float(sites * site + bonds * bond)


def _bytes_site(D, chi, d):
    return 8.0 * (D**4 * d + 4 * chi * chi + 4 * chi * chi * D * D)


def work(case):
    kind = case["kind"]
    if kind == "svd":
        m, k, n, q = case["m"], case["k"], case["n"], case["q"]
        e = {1: m * n, 2: m * k + k * n, 4: m * k + 2 * k * k + k * n}[case["factors"]]
        return {"bytes": 8.0 * (e + (m + 2 * n) * q), "flops": 2.0 * e * q * (2 + 2 * case["niter"])}
    if kind == "als":
        nD, bD, pD = case["nD"], case["bD"], case["pD"]
        one = 2.0 * nD**4 * bD * pD + 2.0 * nD**3 * bD * bD * pD * nD + (nD * bD)**3 / 3
        return {"bytes": 8.0 * (nD**4 + 2 * nD**2 * pD**2),
                "flops": case["iters"] * (2 * one + 2.0 * nD**4 * pD**2)}
    if kind == "sweep":
        b = f = 0.0
        for D, chi in _sweep_sizes(case):
            b += 2 * 4 * _bytes_site(D, chi, case["d"])
            f += 8 * _work_move(D, chi, case["d"], 2, 0, 0, 2, True)
        return {"bytes": b, "flops": f}
    D, chi, d = case["D"], case["chi"], case["d"]
    if kind == "rdm":
        return {"bytes": 2 * _bytes_site(D, chi, d), "flops": _work_rdm(D, chi, d, 1, 1)}
    if kind == "norm":
        nD = case["nD"]
        half = (2 * chi**3 * D**4 + 2 * chi**2 * D**5 * nD + 2 * chi**2 * D**4 * nD * nD
                + 2 * chi**3 * D**2 * nD * nD)
        return {"bytes": 2 * _bytes_site(D, chi, d) + 8.0 * (nD**4 + 2 * D**3 * nD),
                "flops": 2.0 * half + 2.0 * chi * chi * nD**4}
    factors = 4 if case["projectors"] == "full-system" else 2
    q = min(chi + case["over"], chi * D * D)
    nx, ny = case["nx"], case["ny"]
    full_rank = case.get("svd") == "full-rank"
    if kind in ("iterate", "columns"):
        rows = (4 if kind == "iterate" else 2) * nx * ny
    else:
        rows = (ny if case["k"] % 2 == 0 else nx) * (2 if kind == "pair" else 1)
    flops = _work_move(D, chi, d, rows, q, case["niter"], factors, full_rank)
    if kind in ("iterate", "columns"):
        flops += _work_rdm(D, chi, d, nx * ny, 2 * nx * ny)
    else:
        flops += _work_rdm(D, chi, d, len(_written(case)[1]), 0)
    return {"bytes": 2.0 * nx * ny * _bytes_site(D, chi, d), "flops": flops}


# ---------------------------------------------------------------- the same in plain torch, 64 bits
def _exact_als(case, seed):
    nD, bD, pD = case["nD"], case["bD"], case["pD"]
    n12, a12g = _als_inputs(case, seed)
    u, s, vh = torch.linalg.svd(a12g.permute(0, 2, 1, 3).reshape(nD * pD, nD * pD))
    sq = (s[:bD] / s[0]).sqrt()
    a1 = ein("ypu,u->yup", u[:, :bD].reshape(nD, pD, bD), sq)
    a2 = ein("xqv,v->xvq", vh.T[:, :bD].reshape(nD, pD, bD), sq)
    n12g = ein("yxYX,yxpq->YXpq", n12, a12g)

    def solve(r, b):
        r = r.reshape(nD * bD, nD * bD)
        r = (r + r.T) / 2
        r = r + 1e-12 * r.abs().max() * torch.eye(nD * bD, device="cuda", dtype=torch.float64)
        return torch.cholesky_solve(b.reshape(nD * bD, pD), torch.linalg.cholesky(r)).reshape(nD, bD, pD)

    for _ in range(case["iters"]):
        r = ein("yYXuQ,XUQ->YUyu", ein("yxYX,xuq->yYXuq", n12, a2), a2)
        a1 = solve(r, ein("YXpQ,XUQ->YUp", n12g, a2))
        r = ein("xYXvP,YVP->XVxv", ein("yxYX,yvp->xYXvp", n12, a1), a1)
        a2 = solve(r, ein("YXPq,YVP->XVq", n12g, a1))
    return ein("yup,xuq->yxpq", a1, a2)


def exact(case, seed):
    kind = case["kind"]
    torch.manual_seed(seed)
    if kind == "svd":
        mats = _matrices(case, seed)
        torch.manual_seed(seed)
        omega = torch.randn(case["n"], case["q"], dtype=torch.float64, device="cuda")
        return _sign(*_rsvd(mats, case["q"], case["niter"], omega))
    if kind == "als":
        return _exact_als(case, seed)
    if kind == "sweep":
        cfg = dict(projectors="half-system", svd="full-rank")
        out = []
        for i, (D, chi) in enumerate(_sweep_sizes(case)):
            st = _environment(D, chi, case["d"], 2, 2, 0.3, 100 * seed + i)
            for _ in range(2):  # the iteration before the capture, and the pass
                for k, idx in _sweep(2, 2):
                    _move(st, k, idx, 2, 2, chi, cfg, None)
            out.append(_site_rdm(st[0, 0]))
        return out
    nx, ny = case.get("nx", 2), case.get("ny", 2)
    D, chi = case["D"], case["chi"]
    st = _environment(D, chi, case["d"], nx, ny, case.get("bias", 0.0), seed)
    if kind == "rdm":
        s1, s2, k = _bond(case["k"])
        return {"bond": _bond_rdm(st[s1], st[s2], k), "site": _site_rdm(st[0, 1])}
    if kind == "norm":
        g = _generator(seed + 7)
        q = [torch.linalg.qr(_randn(g, D ** 3, case["nD"]))[0].reshape(D, D, D, -1)
             for _ in range(2)]
        s1, s2, k = _bond(case["k"])
        return _norm_tensor(st[s1], st[s2], k, *q)
    if D > 6:
        return None
    torch.manual_seed(seed)

    def omega(n, q):
        return torch.randn(n, q, dtype=torch.float64, device="cuda")

    cfg = dict(projectors=case["projectors"], svd=case.get("svd", "rsvd"), over=case["over"],
               niter=case["niter"])
    if kind in ("iterate", "columns"):
        for k, idx in _sweep(nx, ny)[: 2 * nx if kind == "columns" else None]:
            _move(st, k, idx, nx, ny, chi, cfg, omega)
        bonds = ([((x, y), ((x + 1) % nx, y), 2) for x in range(nx) for y in range(ny)]
                 + [((x, y), (x, (y + 1) % ny), 1) for y in range(ny) for x in range(nx)])
        return {"site": [_site_rdm(st[x, y]) for x in range(nx) for y in range(ny)],
                "bond": [_bond_rdm(st[a], st[b], k) for a, b, k in bonds]}
    moves, sites = _written(case)
    for k, idx in moves:
        _move(st, k, idx, nx, ny, chi, cfg, omega)
    return [_site_rdm(st[s]) for s in sites]
