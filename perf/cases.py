"""The work that users of this package have it do, as measurable cases.

Every case goes through the package's public entry points with the inputs that
a program holds before the call: densities or coefficients made from a seed,
the radial basis, and the handle (batch, bank cache) such a program keeps.
Sizes are those of the package's own workloads (``atomx_b200.workloads``) and
of its tests and benchmark, with ragged ones in between.

``exact`` evaluates the same quantities in 64-bit torch without the package's
kernels: the Gauss-grid Y^k rule as cell sums, the cell algorithm as bank
matrices assembled from cell moments, the trapezoid rule as cumulative sums.
"""
from __future__ import annotations

from functools import lru_cache

import numpy as np
import torch

from atomx_b200 import basis, convol, dirac, quadrature, yk
from atomx_b200.batch import SplitBatch
from atomx_b200.tables import slater_rk_tables, upload_ion
from atomx_b200.workloads import Ion, IonSpec, kappa_ladder

# --------------------------------------------------------------- the cases
_YB = dict(Z=70, ns=120, ks=9, ng=8, r_min=1e-6, r_max=60.0)


def listed():
    return [
        # one screening function on a small ion's grid: the smallest call of
        # the drop-in, latency only (an SCF step makes thousands)
        dict(name="yk_single", kind="yk", rows=1, Z=10, ns=40, ks=7, ng=7, r_min=1e-5, r_max=40.0, k_max=2),
        # a block of densities with mixed multipoles on the Z=70 grid, as a
        # table builder or an MBPT sum forms them
        dict(name="yk_rows", kind="yk", rows=20000, k_max=12, **_YB),
        # the smallest whole table (Z=10, five spinors), plain FP64
        dict(name="table_small", kind="table", precision="fp64", host=False, Z=10, ns=40, ks=7, ng=7, r_min=1e-5,
             r_max=40.0, spinors=5, kappas=2, k_max=2),
        # every R^k of the Z=70 ion, 200 spinors, k <= 12: the scale-up
        # workload, in both precisions
        dict(name="table_fp64", kind="table", precision="fp64", host=False, spinors=200, kappas=7, k_max=12, **_YB),
        dict(name="table_split", kind="table", precision="split", host=False, spinors=200, kappas=7, k_max=12, **_YB),
        # a CI-sized basis (200 splines, 11 nodes per cell, N = 2112): the
        # longest rows, fewer spinors so that the whole table stays on the GPU
        dict(name="table_split_long", kind="table", precision="split", host=False, Z=54, ns=200, ks=9, ng=11,
             r_min=1e-6, r_max=60.0, spinors=160, kappas=9, k_max=16),
        # a ragged mid-size ion, delivered packed to pinned host memory as a
        # CPU-side CI code takes it
        dict(name="table_host", kind="table", precision="split", host=True, Z=37, ns=87, ks=7, ng=7, r_min=1e-5,
             r_max=40.0, spinors=61, kappas=6, k_max=10),
        # many uneven ions in one captured launch (the batch workload's ranges)
        dict(name="batch_uneven", kind="batch", ions=10, draw=3064, max_ns=160, max_spinors=150),
        # cell (bank) integrals by key, as CI/MBPT evaluators request them:
        # a host dict of coefficients in, a list of integrals out
        dict(name="cell_integrals", kind="cell_keys", keys=2000, spinors=40, kappas=5, k_max=8, **_YB),
        # the whole cell table of a 100-spinor ion, banks kept
        dict(name="cell_table", kind="cell_table", spinors=100, kappas=7, k_max=12, **_YB),
        # Dirac-Fock: the DBSR Fock blocks of every occupied subshell, one SCF step
        dict(name="fock_blocks", kind="fock", spinors=24, kappas=4, k_max=7, **_YB),
        # pair potentials on an arbitrary scattering grid, two consumers a row
        dict(name="grid_pair_dots", kind="grid", points=20000, rows=4000, waves=32, consumers=2, k_max=16),
    ]


def _log_int(rng, lo, hi):
    return int(round(float(lo) * (float(hi) / float(lo)) ** rng.random()))


def _draw_basis(rng, most_ns=200):
    ks = rng.choice([7, 9])
    return dict(Z=rng.randint(2, 92), ns=rng.randint(30, most_ns), ks=ks, ng=rng.choice([ks, 8, ks + 2]),
                r_min=rng.choice([1e-6, 1e-5]), r_max=rng.choice([40.0, 60.0]))


def draw(rng):
    kind = rng.choice(["yk", "table", "table", "table", "batch", "cell_keys", "cell_table", "fock", "grid"])
    if kind == "yk":
        return dict(kind=kind, rows=_log_int(rng, 1, 20000), k_max=rng.randint(0, 14), **_draw_basis(rng))
    if kind == "table":
        while True:
            c = dict(kind=kind, precision=rng.choice(["split", "split", "fp64"]), host=rng.random() < 0.2,
                     spinors=_log_int(rng, 4, 200), kappas=rng.randint(1, 7), k_max=rng.randint(2, 14),
                     **_draw_basis(rng))
            if c["host"]:
                c["spinors"] = min(c["spinors"], 80)
            # at most the largest listed table, and no kappa asked for more states than the basis holds
            if _fits(c) and c["spinors"] ** 4 * c["ns"] * c["ng"] * (c["k_max"] + 1) <= 200 ** 4 * 120 * 8 * 13:
                return c
    if kind == "batch":
        return dict(kind=kind, ions=rng.randint(2, 10), draw=rng.randint(1, 9999), max_ns=rng.randint(60, 160),
                    max_spinors=rng.randint(30, 150))
    if kind == "grid":
        return dict(kind=kind, points=_log_int(rng, 300, 20000), rows=_log_int(rng, 10, 4000),
                    waves=rng.randint(4, 32), consumers=rng.randint(1, 4), k_max=rng.randint(0, 16))
    while True:
        c = dict(kind=kind, kappas=rng.randint(1, 7), **_draw_basis(rng, 120))
        if kind == "cell_keys":
            c.update(keys=_log_int(rng, 1, 2000), spinors=rng.randint(4, 40), k_max=rng.randint(0, 8))
        elif kind == "cell_table":
            c.update(spinors=_log_int(rng, 6, 100), k_max=rng.randint(1, 12))
        else:
            c.update(spinors=rng.randint(3, 24), k_max=rng.randint(1, 7))
        if _fits(c):
            return c


def _fits(c):
    """Whether the basis holds the states that one kappa is asked for."""
    return -(-c["spinors"] // (2 * c["kappas"])) <= (c["ns"] - 8) // 2


# -------------------------------------------------------------- the inputs
@lru_cache(maxsize=32)
def _basis(ns, ks, ng, r_min, r_max):
    t = basis.make_exponential_knots(ns, ks, r_min, r_max)
    return basis.prepare_bspline_data(t, ns, ks, n_gauss=ng, kinetic_balance=True)


@lru_cache(maxsize=512)
def _spinors(ns, ks, ng, r_min, r_max, Z, kappa, count):
    """The lowest Dirac-Coulomb spinors of one kappa (not rotated)."""
    P, Q, _ = dirac.dirac_spinors(_basis(ns, ks, ng, r_min, r_max), kappa, Z, count)
    return P, Q


def _shells(spinors, kappas):
    kaps = kappa_ladder(kappas)
    base, extra = divmod(spinors, len(kaps))
    return tuple((kap, base + (i < extra)) for i, kap in enumerate(kaps) if base + (i < extra) > 0)


def _ion(c, seed):
    """The case's ion: the lowest spinors, rotated within each kappa by the seed."""
    key = (c["ns"], c["ks"], c["ng"], c["r_min"], c["r_max"])
    rng = np.random.default_rng(seed)
    P, Q, kap = [], [], []
    for kappa, count in _shells(c["spinors"], c["kappas"]):
        p, q = _spinors(*key, c["Z"], kappa, count)
        if count == 1:  # nothing to rotate: the state of a slightly other mixture, so that seeds differ
            p2, q2 = _spinors(*key, c["Z"], kappa, 2)
            th = 0.2 * rng.standard_normal()
            rot = np.array([[np.cos(th), np.sin(th)]])
            p, q = rot @ p2, rot @ q2
        else:
            rot, r = np.linalg.qr(rng.standard_normal((count, count)))
            rot = (rot * np.sign(np.diag(r))[None, :]).T
            p, q = rot @ p, rot @ q
        P.append(p)
        Q.append(q)
        kap += [kappa] * count
    spec = IonSpec(Z=c["Z"], ns=c["ns"], ks=c["ks"], n_gauss=c["ng"], r_min=c["r_min"], r_max=c["r_max"],
                   shells=_shells(c["spinors"], c["kappas"]), k_max=c["k_max"], seed=int(seed))
    return Ion(spec=spec, bsp=_basis(*key), P=np.ascontiguousarray(np.concatenate(P)),
               Q=np.ascontiguousarray(np.concatenate(Q)), kappa=np.asarray(kap, dtype=np.int64))


def _batch_cases(c):
    """The ions of an uneven batch (sizes from the case, not from the seed)."""
    rng = np.random.default_rng(c["draw"])
    out = []
    for _ in range(c["ions"]):
        ks = int(rng.choice([7, 9]))
        out.append(dict(Z=int(rng.integers(20, 84)), ns=int(rng.integers(40, c["max_ns"] + 1)), ks=ks, ng=ks,
                        r_min=1e-5, r_max=40.0, spinors=int(rng.integers(20, c["max_spinors"] + 1)), kappas=6,
                        k_max=12))
    return out


def _densities(c, seed):
    """(rows, N) sign-changing Slater-type densities and their multipoles."""
    bd = _basis(c["ns"], c["ks"], c["ng"], c["r_min"], c["r_max"])
    g = torch.Generator().manual_seed(int(seed))
    rows = c["rows"]
    zeta = 0.5 * torch.exp(torch.rand(rows, 1, generator=g, dtype=torch.float64) * float(np.log(4.0 * c["Z"])))
    power = torch.randint(1, 5, (rows, 1), generator=g).to(torch.float64)
    phase = 6.28 * torch.rand(rows, 1, generator=g, dtype=torch.float64)
    r = torch.as_tensor(bd["gr"].reshape(1, -1), device="cuda")
    x = zeta.cuda() * r
    rho = x ** power.cuda() * torch.exp(-x) * torch.cos(x + phase.cuda())
    ks = torch.randint(0, c["k_max"] + 1, (rows,), generator=g).numpy().astype(np.int32)
    return bd, rho, ks


def _grid_inputs(c, seed):
    """Waves, pair rows and consumer weights on a geometric radial grid."""
    rng = np.random.default_rng(seed)
    n, rows = c["points"], c["rows"]
    r = np.geomspace(1e-4, 80.0, n)
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    env = torch.as_tensor(np.exp(-r / 10.0), device="cuda")

    def waves(count):
        return torch.randn(count, n, generator=g, device="cuda", dtype=torch.float64) * env

    PA, QA, PB, QB = waves(c["waves"]), 0.02 * waves(c["waves"]), waves(c["waves"]), 0.02 * waves(c["waves"])
    ptr = np.arange(0, c["consumers"] * rows + 1, c["consumers"])
    return dict(PA=PA, QA=QA, PB=PB, QB=QB, a=rng.integers(0, c["waves"], rows), b=rng.integers(0, c["waves"], rows),
                k=rng.integers(0, c["k_max"] + 1, rows), ok=np.ones(rows, dtype=bool), W=waves(8), ptr=ptr,
                cons=rng.integers(0, 8, c["consumers"] * rows), r=r)


def _keys(c, ion, seed):
    rng = np.random.default_rng(seed + 1)
    n = ion.n_orbitals
    return [(int(a), int(b), int(d), int(e), int(k)) for a, b, d, e, k in
            zip(*(rng.integers(0, n, c["keys"]) for _ in range(4)), rng.integers(0, c["k_max"] + 1, c["keys"]))]


def _angular(c, ion, seed):
    """Angular coefficients with the selection rules of a Dirac-Fock step."""
    rng = np.random.default_rng(seed + 2)
    n = ion.n_orbitals
    ad, ax = np.zeros((n, n, c["k_max"] + 1)), np.zeros((n, n, c["k_max"] + 1))
    for i in range(n):
        for j in range(n):
            ki, kj = int(ion.kappa[i]), int(ion.kappa[j])
            for k in _allowed(ki, kj):
                if k <= c["k_max"]:
                    ax[i, j, k] = -rng.random()
            for k in range(0, min(c["k_max"], 2 * min(abs(ki), abs(kj)) - 1) + 1, 2):
                ad[i, j, k] = 2.0 + rng.random() if k == 0 else -0.1 * rng.random()
    return ad, ax, 1.0 + rng.random(n)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "yk":
        bd, rho, ks = _densities(case, seed)
        gr, grw = torch.as_tensor(bd["gr"], device="cuda"), torch.as_tensor(bd["grw"], device="cuda")
        return dict(case=case, rho=rho, ks=ks, gr=gr, grw=grw)
    if kind == "table":
        return dict(case=case, ion=_ion(case, seed))
    if kind == "batch":
        devs = [upload_ion(_ion(c, seed + i)) for i, c in enumerate(_batch_cases(case))]
        b = SplitBatch(devs)
        b.capture()
        return dict(case=case, batch=b)
    if kind == "grid":
        return dict(case=case, **_grid_inputs(case, seed))
    ion = _ion(case, seed)
    cache = convol.ConvolCache(ion.bsp)
    for k in range(case["k_max"] + 1):
        cache.bank(k)
    st = dict(case=case, ion=ion, cache=cache)
    if kind == "cell_keys":
        st["orbitals"] = {i: (ion.P[i], ion.Q[i]) for i in range(ion.n_orbitals)}
        st["keys"] = _keys(case, ion, seed)
    elif kind == "fock":
        st["angular"] = _angular(case, ion, seed)
    return st


# ---------------------------------------------------------------- the calls
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "yk":
        gr, grw = state["gr"], state["grw"]
        nv, ng = gr.shape
        if case["rows"] == 1:
            return yk.compute_yk(state["rho"].view(nv, ng), gr, grw, nv, ng, int(state["ks"][0]))
        return yk.compute_yk_rows(state["rho"], state["ks"], gr, grw)
    if kind == "table":
        opts = dict(host=True, packed=True) if case["host"] else {}
        return slater_rk_tables(state["ion"], precision=case["precision"], **opts).values
    if kind == "batch":
        b = state["batch"]
        b.replay()
        b.check_status()
        return b.out
    if kind == "cell_keys":
        return np.array(convol.compute_slater_rk_cell_batch(state["orbitals"], state["keys"], state["ion"].bsp,
                                                            state["cache"]))
    if kind == "cell_table":
        ion = state["ion"]
        return convol.cell_tables(ion.P, ion.Q, ion.kappa, ion.bsp, case["k_max"], cache=state["cache"]).values
    if kind == "fock":
        ion = state["ion"]
        ad, ax, norms = state["angular"]
        return convol.build_hf_matrices_dbsr(np.arange(ion.n_orbitals), ion.P, ion.Q, ad, ax,
                                             range(case["k_max"] + 1), norms, ion.bsp, state["cache"])
    s = state
    return quadrature.yk_pair_dot_batch_on_grid(s["PA"], s["QA"], s["PB"], s["QB"], s["a"], s["b"], s["k"], s["ok"],
                                                s["W"], s["ptr"], s["cons"], s["r"])


# ------------------------------------------------- what a pass cannot do without
def _table_work(c):
    n = (c["ns"] - c["ks"] + 1) * c["ng"]
    sizes = [len(p) for _, p in _plan(_kappas(c), c["k_max"])]
    unique, full = sum(m * (m + 1) // 2 for m in sizes), sum(m * m for m in sizes)
    return dict(bytes=8.0 * (unique if c.get("host") else full) + 16.0 * c["spinors"] * c["ns"],
                flops=2.0 * n * unique + 4.0 * n * c["ng"] * sum(sizes))


def work(case):
    c, kind = case, case["kind"]
    if kind == "yk":
        n = (c["ns"] - c["ks"] + 1) * c["ng"]
        return dict(bytes=16.0 * c["rows"] * n, flops=4.0 * c["rows"] * n * c["ng"])
    if kind == "table":
        return _table_work(c)
    if kind == "batch":
        w = [_table_work(x) for x in _batch_cases(c)]
        return dict(bytes=sum(x["bytes"] for x in w), flops=sum(x["flops"] for x in w))
    if kind == "grid":
        return dict(bytes=8.0 * c["points"] * (4 * c["waves"] + 8 + 2 * (c["k_max"] + 1)),
                    flops=c["rows"] * c["points"] * (20.0 + 2.0 * c["consumers"]))
    ns, ks = c["ns"], c["ks"]
    kdim = ns * (2 * ks - 1)
    bank = 8.0 * kdim * kdim
    if kind == "cell_keys":
        # each distinct pair's potential against its multipole's bank, one dot a key
        pairs = min(c["keys"], c["spinors"] ** 2 * (c["k_max"] + 1))
        return dict(bytes=bank * min(c["keys"], c["k_max"] + 1), flops=2.0 * pairs * kdim * kdim)
    if kind == "cell_table":
        sizes = [len(p) for _, p in _plan(_kappas(c), c["k_max"])]
        return dict(bytes=8.0 * sum(m * m for m in sizes) + bank * len(sizes),
                    flops=sum(2.0 * m * kdim * kdim + kdim * m * (m + 1.0) for m in sizes))
    blocks = 4 * (c["k_max"] + 1)
    return dict(bytes=bank * (c["k_max"] + 1) + 32.0 * c["spinors"] * ns * ns,
                flops=blocks * c["spinors"] * 2.0 * ns * ns * (2 * ks) ** 2)


# --------------------------------------------------------- the same in 64 bits
def _allowed(ka, kb):
    la, lb = (k if k > 0 else -k - 1 for k in (ka, kb))
    lo, hi = abs(abs(ka) - abs(kb)), abs(ka) + abs(kb) - 1
    return [k for k in range(lo, hi + 1) if (k + la + lb) % 2 == 0]


def _kappas(c):
    return tuple(kap for kap, n in _shells(c["spinors"], c["kappas"]) for _ in range(n))


@lru_cache(maxsize=16)
def _plan(kappa, k_max):
    """[(k, pairs)] of every allowed multipole: the pairs a <= c that allow k,
    grouped by the shells of a and c."""
    shells, start = [], 0
    for i in range(1, len(kappa) + 1):
        if i == len(kappa) or kappa[i] != kappa[start]:
            shells.append((kappa[start], range(start, i)))
            start = i
    out = {}
    for i, (ka, ra) in enumerate(shells):
        for kc, rc in shells[i:]:
            pairs = [(a, c) for a in ra for c in rc if a <= c]
            for k in _allowed(ka, kc):
                if k <= k_max:
                    out.setdefault(k, []).extend(pairs)
    return [(k, np.asarray(out[k])) for k in sorted(out)]


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _partials(ng):
    """The integral of each Lagrange basis polynomial of a cell up to each node, over its weight."""
    x, _ = np.polynomial.legendre.leggauss(ng)
    P = np.polynomial.legendre.legvander(x, ng)
    prim = np.stack([x + 1] + [(P[:, m + 1] - P[:, m - 1]) / (2 * m + 1) for m in range(1, ng)], axis=1)
    return (prim * ((2 * np.arange(ng) + 1) / 2)) @ P[:, :ng].T


def _yk_exact(g, ks, gr):
    """Y^k of the rows g = w rho (rows, N); ks: one multipole or one a row."""
    nv, ng = gr.shape
    r = torch.as_tensor(gr, device=g.device).reshape(1, nv, ng)
    k = torch.as_tensor(np.asarray(ks, dtype=np.float64), device=g.device).reshape(-1, 1, 1)
    mo = torch.as_tensor(_partials(ng), device=g.device)
    rk, ri = r ** k, r ** (-(k + 1))
    h, e = g.view(-1, nv, ng) * rk, g.view(-1, nv, ng) * ri
    hs, es = h.sum(-1), e.sum(-1)
    a = torch.nn.functional.pad(hs.cumsum(1)[:, :-1], (1, 0))
    b = torch.nn.functional.pad(es.flip(1).cumsum(1)[:, :-1], (1, 0)).flip(1)
    y = ri * (a[..., None] + h @ mo.T) + rk * (b[..., None] + e @ (1 - mo).T)
    return y.reshape(g.shape)


def _values(coef, b):
    nv, ng, ks = b.shape
    idx = np.arange(nv)[:, None] + np.arange(ks)[None, :]
    pad = np.pad(coef, ((0, 0), (0, max(0, nv + ks - 1 - coef.shape[1]))))
    return np.einsum("ovs,vms->ovm", pad[:, idx], b).reshape(coef.shape[0], -1)


def _tables_exact(ion, k_max, packed=False):
    d = _device()
    bd = ion.bsp
    P = torch.as_tensor(_values(ion.P, bd["bsp_p"]), device=d)
    Q = torch.as_tensor(_values(ion.Q, bd["bsp_q"]), device=d)
    w = torch.as_tensor(bd["grw"].reshape(1, -1), device=d)
    out = []
    for k, pairs in _plan(tuple(ion.kappa.tolist()), k_max):
        a, c = torch.as_tensor(pairs[:, 0], device=d), torch.as_tensor(pairs[:, 1], device=d)
        g = w * (P[a] * P[c] + Q[a] * Q[c])
        T = g @ _yk_exact(g, k, bd["gr"]).T
        if packed:
            i, j = torch.triu_indices(T.shape[0], T.shape[0], device=d)
            T = T[i, j]
        out.append(T.reshape(-1))
    return torch.cat(out)


def _spline_values(t, order, x, left):
    """The `order` nonzero B-splines at each x of the interval that starts at knot left (Cox-de Boor)."""
    b = np.zeros(x.shape + (order,))
    b[..., 0] = 1.0
    for j in range(1, order):
        carry = np.zeros(x.shape)
        for i in range(j):
            right, lo = t[left + i + 1], t[left + 1 - (j - i)]
            f = b[..., i] / (right - lo)
            b[..., i] = carry + (right - x) * f
            carry = (x - lo) * f
        b[..., j] = carry
    return b


def _cell_pairs(order):
    return [(h, hp) for h in range(order) for hp in range(h, order)]


def _products(b):
    h = np.array(_cell_pairs(b.shape[-1]))
    return b[..., h[:, 0]] * b[..., h[:, 1]]


@lru_cache(maxsize=24)
def _bank_exact(key, k):
    """{(left, right): (ks_l, ns, ks_r, ns)} bank matrices of one multipole on the device."""
    bd = _basis(*key)
    nv, ns, gr, grw = bd["nv"], bd["ns"], bd["gr"], bd["grw"]
    comp = {"p": (bd["bsp_p"], bd["tp"], bd["ksp"]), "q": (bd["bsp_q"], bd["t"], bd["ksq"])}
    prod = {c: _products(v[0]) for c, v in comp.items()}  # (nv, ng, pairs)
    rise = {c: np.einsum("vm,vmp->vp", grw * gr ** k, prod[c]) for c in comp}
    fall = {c: np.einsum("vm,vmp->vp", grw / gr ** (k + 1), prod[c]) for c in comp}

    def inner_outer(outer, inner, n_sub):
        """[cell][outer pair][inner pair]: the inner electron inside the outer one, both in the cell."""
        _, t, order = comp[inner]
        x, w = np.polynomial.legendre.leggauss(n_sub)
        x, w = 0.5 * (x + 1), 0.5 * w
        res = np.empty((nv, prod[outer].shape[-1], prod[inner].shape[-1]))
        for v in range(nv):
            left = order - 1 + v
            span = (gr[v] - t[left])[:, None]
            gx = t[left] + span * x[None, :]
            b = _products(_spline_values(t, order, gx, left))
            acc = np.einsum("mn,mnp->mp", span * w[None, :] * gx ** k, b)
            res[v] = np.einsum("m,mo,mp->op", grw[v] / gr[v] ** (k + 1), prod[outer][v], acc)
        return res

    d = _device()
    up = torch.triu(torch.ones(nv, nv, dtype=torch.float64, device=d), 1)
    out = {}
    for lc, rc in (("p", "p"), ("q", "q"), ("p", "q"), ("q", "p")):
        ksl, ksr = comp[lc][2], comp[rc][2]
        n_sub = max(ksl, ksr) + k // 2
        dia = inner_outer(lc, rc, n_sub) + inner_outer(rc, lc, n_sub).transpose(0, 2, 1)
        rl, fl, rr, fr = (torch.as_tensor(x, device=d) for x in (rise[lc], fall[lc], rise[rc], fall[rc]))
        pl, pr = _cell_pairs(ksl), _cell_pairs(ksr)
        # A[pl, v, pr, u], then folded onto the global pairs (s, i) of both sides
        A = (torch.einsum("vp,uq,vu->pvqu", rl, fr, up) + torch.einsum("vp,uq,uv->pvqu", fl, rr, up))
        i = torch.arange(nv, device=d)
        A[:, i, :, i] += torch.as_tensor(dia, device=d)
        K1 = torch.zeros(ksl, ns, len(pr), nv, dtype=torch.float64, device=d)
        for p, (h, hp) in enumerate(pl):
            K1[hp - h, h:h + nv] += A[p]
        K = torch.zeros(ksl, ns, ksr, ns, dtype=torch.float64, device=d)
        for q, (h, hp) in enumerate(pr):
            K[:, :, hp - h, h:h + nv] += K1[:, :, q]
        out[lc, rc] = K
    return out


def _bands(C, pairs, ks):
    """Banded pair densities (n, ks, ns) of the coefficient rows C."""
    a, b = C[pairs[:, 0]], C[pairs[:, 1]]
    ns = C.shape[1]
    D = torch.zeros(len(pairs), ks, ns, dtype=C.dtype, device=C.device)
    D[:, 0] = a * b
    for s in range(1, ks):
        D[:, s, :ns - s] = a[:, :ns - s] * b[:, s:] + a[:, s:] * b[:, :ns - s]
    return D


def _basis_key(c):
    return (c["ns"], c["ks"], c["ng"], c["r_min"], c["r_max"])


def _potential_rows(bank, dp, dq):
    """The potentials (P and Q bands) of densities with bands dp, dq."""
    return (torch.einsum("siuj,nuj->nsi", bank["p", "p"], dp) + torch.einsum("siuj,nuj->nsi", bank["p", "q"], dq),
            torch.einsum("siuj,nuj->nsi", bank["q", "p"], dp) + torch.einsum("siuj,nuj->nsi", bank["q", "q"], dq))


def _coefficients(ion):
    d = _device()
    return torch.as_tensor(ion.P, device=d), torch.as_tensor(ion.Q, device=d)


def _cell_table_exact(c, ion):
    P, Q = _coefficients(ion)
    ksp, ksq = ion.bsp["ksp"], ion.bsp["ksq"]
    out = []
    for k, pairs in _plan(tuple(ion.kappa.tolist()), c["k_max"]):
        pr = torch.as_tensor(pairs, device=P.device)
        dp, dq = _bands(P, pr, ksp), _bands(Q, pr, ksq)
        wp, wq = _potential_rows(_bank_exact(_basis_key(c), k), dp, dq)
        n = len(pairs)
        out.append((dp.reshape(n, -1) @ wp.reshape(n, -1).T + dq.reshape(n, -1) @ wq.reshape(n, -1).T).reshape(-1))
    return torch.cat(out)


def _cell_keys_exact(c, ion, seed):
    P, Q = _coefficients(ion)
    ksp, ksq = ion.bsp["ksp"], ion.bsp["ksq"]
    keys = np.array(_keys(c, ion, seed))
    out = torch.zeros(len(keys), dtype=torch.float64, device=P.device)
    for k in sorted(set(keys[:, 4].tolist())):
        at = torch.as_tensor(np.flatnonzero(keys[:, 4] == k), device=P.device)
        kk = torch.as_tensor(keys, device=P.device)[at]
        wp, wq = _potential_rows(_bank_exact(_basis_key(c), k), _bands(P, kk[:, 2:4], ksp), _bands(Q, kk[:, 2:4], ksq))
        out[at] = (_bands(P, kk[:, :2], ksp) * wp).sum((1, 2)) + (_bands(Q, kk[:, :2], ksq) * wq).sum((1, 2))
    return out.cpu().numpy()


def _fock_exact(c, ion, seed):
    ad, ax, norms = _angular(c, ion, seed)
    C = dict(zip("pq", _coefficients(ion)))
    d, n, ns = C["p"].device, ion.n_orbitals, ion.bsp["ns"]
    ad, ax = torch.as_tensor(ad, device=d), torch.as_tensor(ax, device=d)
    H = {x: torch.zeros(n, ns, ns, dtype=torch.float64, device=d) for x in ("pp", "qq", "pq", "qp")}
    order = {"p": ion.bsp["ksp"], "q": ion.bsp["ksq"]}
    own = torch.arange(n, device=d)
    for k in range(c["k_max"] + 1):
        bank = _bank_exact(_basis_key(c), k)
        co = ad[:, :, k].clone()
        co[own, own] *= 2.0
        for x in "pq":
            for y in "pq":
                K = bank[x, y]
                self_bands = _bands(C[y], torch.stack([own, own], 1), order[y])
                v = torch.einsum("siuj,nuj->nsi", K, torch.einsum("nm,muj->nuj", co, self_bands))
                for s in range(order[x]):
                    h = H[x + x]
                    i = torch.arange(ns - s, device=d)
                    h[:, i, i + s] += v[:, s, :ns - s]
                    if s:
                        h[:, i + s, i] += v[:, s, :ns - s]
                dens = torch.einsum("nm,mi,mj->nij", ax[:, :, k], C[x], C[y])
                for di in range(1 - order[x], order[x]):
                    rows = torch.arange(max(0, -di), min(ns, ns - di), device=d)
                    for dj in range(1 - order[y], order[y]):
                        cols = torch.arange(max(0, -dj), min(ns, ns - dj), device=d)
                        G = K[abs(di)][torch.minimum(rows, rows + di)][:, abs(dj)][:, torch.minimum(cols, cols + dj)]
                        H[x + y][:, rows[0]:rows[-1] + 1, cols[0]:cols[-1] + 1] += \
                            G * dens[:, rows[0] + di:rows[-1] + di + 1, cols[0] + dj:cols[-1] + dj + 1]
    pq = 0.5 * (H["pq"] + H["qp"].transpose(1, 2))
    out = torch.stack([0.5 * (H["pp"] + H["pp"].transpose(1, 2)), 0.5 * (H["qq"] + H["qq"].transpose(1, 2)), pq,
                       pq.transpose(1, 2)], dim=1)
    return out / torch.as_tensor(norms, device=d).reshape(-1, 1, 1, 1)


def _grid_exact(c, seed):
    s = _grid_inputs(c, seed)
    d = s["PA"].device
    r = torch.as_tensor(s["r"], device=d)
    dr = r[1:] - r[:-1]
    a, b, kk = (torch.as_tensor(s[x], device=d) for x in ("a", "b", "k"))
    cons = torch.as_tensor(s["cons"], device=d).view(-1, c["consumers"])
    out = torch.empty(cons.shape, dtype=torch.float64, device=d)
    for lo in range(0, c["rows"], 512):
        at = slice(lo, lo + 512)
        rho = s["PA"][a[at]] * s["PB"][b[at]] + s["QA"][a[at]] * s["QB"][b[at]]
        k = kk[at].to(torch.float64)[:, None]
        up, down = r[None, :] ** k, r[None, :] ** (-(k + 1))
        f, g = rho * up, rho * down
        zero = torch.zeros(f.shape[0], 1, dtype=torch.float64, device=d)
        inner = torch.cat([zero, (0.5 * (f[:, 1:] + f[:, :-1]) * dr).cumsum(1)], 1)
        outer = torch.cat([(0.5 * (g[:, 1:] + g[:, :-1]) * dr).flip(1).cumsum(1).flip(1), zero], 1)
        y = inner * down + up * outer
        out[at] = torch.einsum("rci,ri->rc", s["W"][cons[at]], y)
    return out.reshape(-1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "yk":
        bd, rho, ks = _densities(case, seed)
        g = rho * torch.as_tensor(bd["grw"].reshape(1, -1), device=rho.device)
        if case["rows"] == 1:
            return _yk_exact(g, int(ks[0]), bd["gr"]).view(bd["gr"].shape)
        return torch.cat([_yk_exact(g[i:i + 2048], ks[i:i + 2048], bd["gr"]) for i in range(0, len(ks), 2048)])
    if kind == "table":
        v = _tables_exact(_ion(case, seed), case["k_max"], packed=case["host"])
        return v.cpu() if case["host"] else v
    if kind == "batch":
        return torch.cat([_tables_exact(_ion(c, seed + i), c["k_max"]) for i, c in enumerate(_batch_cases(case))])
    if kind == "grid":
        return _grid_exact(case, seed)
    ion = _ion(case, seed)
    if kind == "cell_keys":
        return _cell_keys_exact(case, ion, seed)
    return _cell_table_exact(case, ion) if kind == "cell_table" else _fock_exact(case, ion, seed)
