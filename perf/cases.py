"""What a user has this library do, as measurable cases: one entry point each,
at the sizes of the benchmark configurations, the mode trees and the learned
warm start.

A case is a dict of plain values; ``kind`` names the entry point:

* ``als``       ``als.reduce_batched`` on device-resident vectors, or, with
                ``host``, one ``alscpp`` call on host arrays (the Fortran host);
* ``cycle``     ``intertwine.intertwine``: power sweeps, Gram-Schmidt and, with
                ``update``, the Rayleigh-Ritz step and the vector updates;
* ``range``     ``intertwine.spectral_range`` from the solver's starting vectors;
* ``rayleigh``  ``intertwine.qhq_diag``, the ``update = F`` step;
* ``carry``     ``intertwine.qhq`` with a one-term operator list: a coupling
                carried into a solved node's basis (mode trees);
* ``diag``      ``intertwine.diagonalize`` of a two-mode node whose block is every
                product function;
* ``svd``       ``intertwine.reduc_svd``, the two-mode reduction;
* ``mlp``       one training step of the warm start's network.

The launch-shape searches are switched off (``mlcp_gb300_set_autotune``), so that
a case runs the same launch shapes, and gives the same bits, in every process.
``exact`` restates each computation in 64 bits from its definition.
"""
import math

import numpy as np
import torch

from mlcp_gb300 import _lib, als, hoplist, intertwine, solver, workloads
from mlcp_gb300.mlp import Mlp


def listed():
    return [
        # the ALS microbenchmark: the power step of a 30-mode block, rank 20 x 160 terms back to rank 20
        {"name": "als_block_64x30", "kind": "als", "nvec": 64, "modes": 30, "n_lo": 12, "n_hi": 12, "rank": 20,
         "target": 3200, "sweeps": 10, "host": False},
        # one reduction as the Fortran host calls it: a Henon-Heiles power step, rank 16 x (11 terms + shift)
        {"name": "als_host_1x6", "kind": "als", "nvec": 1, "modes": 6, "n_lo": 10, "n_hi": 10, "rank": 16,
         "target": 192, "sweeps": 10, "host": True},
        # the Gram-Schmidt of the benchmark's power cycle by itself: 40 states, rank 16, psinals 10
        {"name": "ortho_hh6_40", "kind": "cycle", "ham": "hh", "modes": 6, "n_lo": 10, "n_hi": 10, "terms": 0,
         "block": 40, "rank": 16, "rank_lo": 16, "npow": 0, "nals": 10, "update": False},
        # one cycle of a tree's top node over three groups of 30 states
        {"name": "cycle_top3_40", "kind": "cycle", "ham": "qff", "modes": 3, "n_lo": 30, "n_hi": 30, "terms": 0,
         "block": 40, "rank": 16, "rank_lo": 16, "npow": 2, "nals": 2, "update": True},
        # one sweep of everything on the largest node: six groups of 48 states, 100 states, rank 30, hundreds of terms
        {"name": "cycle_top6_100", "kind": "cycle", "ham": "random", "modes": 6, "n_lo": 48, "n_hi": 48, "terms": 400,
         "block": 100, "rank": 30, "rank_lo": 30, "npow": 1, "nals": 1, "update": True},
        # ragged ranks 8-64 over uneven bases of 4-10 functions: power sweep and Gram-Schmidt
        {"name": "ragged_12x32", "kind": "cycle", "ham": "qff", "modes": 12, "n_lo": 4, "n_hi": 10, "terms": 0,
         "block": 32, "rank": 64, "rank_lo": 8, "npow": 1, "nals": 1, "update": False},
        # the spectral range before every node's solve: its first two rounds, five power steps each on two vectors
        {"name": "range_hh6", "kind": "range", "ham": "hh", "modes": 6, "n_lo": 10, "n_hi": 10, "terms": 0, "rank": 16,
         "npow": 5, "rounds": 2},
        # Rayleigh quotients of the benchmark's block: the smallest call
        {"name": "rayleigh_hh6_40", "kind": "rayleigh", "ham": "hh", "modes": 6, "n_lo": 10, "n_hi": 10, "terms": 0,
         "block": 40, "rank": 16},
        # a coupling carried into the basis of a solved group node (two pairs of 24 states, 48 states kept)
        {"name": "carry_24x24_48", "kind": "carry", "modes": 2, "n_lo": 24, "n_hi": 24, "block": 48, "rank": 24},
        # the exact solution of a two-mode node: all 12 x 12 product functions, a new Hamiltonian each time
        {"name": "diag_12x12", "kind": "diag", "n": 12, "rank": 8},
        # the two-mode reduction of 64 power-step vectors: 21 x 16 terms on a 40 x 40 basis to rank 16
        {"name": "svd_64x40x40", "kind": "svd", "nvec": 64, "nr": 40, "nc": 40, "terms": 336, "rank": 16},
        # one training step of the warm start: 24 vectors x 6 modes x 5 cycles, bases of 8 functions, rank 30
        {"name": "mlp_train_720", "kind": "mlp", "rows": 720, "n": 8, "rank": 30},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["als", "als", "cycle", "cycle", "cycle", "ragged", "range", "rayleigh", "carry", "diag", "svd",
                       "mlp"])
    if kind == "als":
        host = rng.random() < 0.3
        n = _log(rng, 8, 24)
        return {"kind": kind, "nvec": 1 if host else _log(rng, 1, 64), "modes": _log(rng, 8, 30),
                "n_lo": max(6, n - rng.randint(0, 5)), "n_hi": n, "rank": (r := rng.randint(4, 32)),
                "target": _log(rng, 16 * r, 3200), "sweeps": rng.randint(1, 4), "host": host}
    if kind == "cycle":
        ortho = rng.random() < 0.5
        n, modes = _log(rng, 12, 48), rng.randint(3, 6)
        ham = rng.choice(["qff", "random"])
        return {"kind": kind, "ham": ham, "modes": modes, "n_lo": n - rng.randint(0, 4), "n_hi": n,
                "terms": _log(rng, 20, 400), "block": _log(rng, 12, 100), "rank": (r := rng.randint(8, 30)), "rank_lo": r,
                "npow": 0 if ortho else 1, "nals": rng.randint(1, 2) if ortho else 1, "update": not ortho}
    if kind == "ragged":
        r = rng.randint(12, 64)
        return {"kind": "cycle", "ham": "qff", "modes": rng.randint(6, 12), "n_lo": 4, "n_hi": rng.randint(7, 10),
                "terms": 0, "block": _log(rng, 6, 32), "rank": r, "rank_lo": 8, "npow": 1, "nals": 1, "update": False}
    if kind == "range":
        n = _log(rng, 8, 24)
        return {"kind": kind, "ham": "hh", "modes": rng.randint(5, 8), "n_lo": n, "n_hi": n, "terms": 0,
                "rank": rng.randint(8, 20), "npow": rng.randint(2, 5), "rounds": rng.randint(1, 2)}
    if kind == "rayleigh":
        n = _log(rng, 6, 48)
        return {"kind": kind, "ham": rng.choice(["hh", "qff"]), "modes": rng.randint(3, 8), "n_lo": n, "n_hi": n,
                "terms": 0, "block": _log(rng, 4, 100), "rank": rng.randint(4, 32)}
    if kind == "carry":
        n = _log(rng, 8, 48)
        return {"kind": kind, "modes": rng.randint(2, 3), "n_lo": n - rng.randint(0, 3), "n_hi": n,
                "block": _log(rng, 10, 100), "rank": rng.randint(6, 30)}
    if kind == "diag":
        n = rng.randint(5, 12)
        return {"kind": kind, "n": n, "rank": rng.randint(3, 2 * n // 3)}
    if kind == "svd":
        return {"kind": kind, "nvec": _log(rng, 1, 64), "nr": _log(rng, 8, 64), "nc": _log(rng, 8, 64),
                "terms": _log(rng, 16, 400), "rank": rng.randint(4, 24)}
    return {"kind": kind, "rows": _log(rng, 100, 2000), "n": rng.randint(5, 12), "rank": rng.randint(8, 30)}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------

def _bases(case):
    """Basis sizes: n_lo .. n_hi, the same in every state of a case."""
    rng = np.random.default_rng(case["modes"])
    nb = rng.integers(case["n_lo"], case["n_hi"] + 1, case["modes"])
    nb[0] = case["n_hi"]
    return [int(x) for x in nb]


def _operators(case):
    """The node's operator list: one Hamiltonian for all of a case's states, as a solver keeps it over its cycles."""
    nb = _bases(case)
    if case["ham"] == "hh":
        return hoplist.henon_heiles(case["modes"], case["n_hi"])
    if case["ham"] == "qff":
        return hoplist.synthetic_qff(case["modes"], nb, 5, cubic_frac=0.3 if case["modes"] < 10 else 0.1)
    return hoplist.random_hoplist(nb, case["terms"], 7)


def _block(case, rng, nb):
    """A block of random CP vectors (the reference's starting guess): factors uniform in [-0.5, 0.5), weights 1."""
    rows = case["block"] * case["rank"]
    return rng.uniform(-0.5, 0.5, size=(rows, sum(nb))), np.ones(rows)


def _inputs(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "als":
        b = workloads.als_batch(case["nvec"], case["modes"], _bases(case), case["rank"], case["target"], seed=seed)
        return {"batch": b}
    if kind in ("cycle", "rayleigh"):
        hl = _operators(case)
        base, coef = _block(case, rng, hl.nbas)
        ranks = None
        if kind == "cycle" and case["rank_lo"] < case["rank"]:
            ranks = np.random.default_rng(case["block"]).integers(case["rank_lo"], case["rank"] + 1, case["block"])
        shift = {"hh": 5.0 * case["modes"], "qff": 20000.0, "random": 33.0}[case["ham"]]
        return {"hl": hl, "base": base, "coef": coef, "ranks": ranks, "shift": shift}
    if kind == "range":
        hl = _operators(case)
        base, coef = solver.spectral_start(hl.nbas, case["rank"], seed)
        return {"hl": hl, "base": base, "coef": coef}
    if kind == "carry":
        nb = _bases(case)
        g = np.random.default_rng(3)
        ops = {d: (m + m.T) for d, m in ((d, g.normal(size=(n, n)) / math.sqrt(n)) for d, n in enumerate(nb))}
        base, coef = _block(case, rng, nb)
        return {"hl": hoplist.build_hoplist(nb, [(1.0, ops)]), "base": base, "coef": coef}
    if kind == "diag":
        n, rk = case["n"], case["rank"]
        # cubic constants of its own for each state; no two levels of this force field are nearly degenerate, so its
        # eigenvectors have values to compare
        hl = hoplist.synthetic_qff(2, n, 34, cubic_sigma=50.0 * rng.uniform(0.9, 1.1))
        base, coef = np.zeros((n * n * rk, 2 * n)), np.zeros(n * n * rk)
        for a in range(n):
            for b in range(n):
                base[(a * n + b) * rk, [a, n + b]] = 1.0
                coef[(a * n + b) * rk] = 1.0
        return {"hl": hl, "base": base, "coef": coef}
    if kind == "svd":
        rows = case["nvec"] * case["terms"]
        return {"base": rng.normal(size=(rows, case["nr"] + case["nc"])), "coef": rng.uniform(0.1, 1.0, rows)}
    ins, outs = 64 * (case["n"] + 1), case["n"] * case["rank"]
    x = rng.normal(size=(case["rows"], ins)) / math.sqrt(case["n"])
    t = rng.normal(size=(case["rows"], outs)) / math.sqrt(case["n"])
    return {"x": x.astype(np.float32), "t": t.astype(np.float32)}


def prepare(case, seed):
    lib = _lib.load()
    lib.mlcp_gb300_set_autotune(0)
    s = _inputs(case, seed)
    s["case"] = case
    if case["kind"] == "als":
        b = s["batch"]
        if case["host"]:
            s["start"] = b.coef[:case["rank"]].copy(), b.base[:case["rank"]].copy()
        else:
            dev = torch.device("cuda", torch.cuda.current_device())
            s["coef"], s["base"] = torch.from_numpy(b.coef).to(dev), torch.from_numpy(b.base).to(dev)
            f, each = case["rank"], case["rank"] + case["target"]
            s["F"] = s["coef"].view(b.nvec, each)[:, :f], s["base"].view(b.nvec, each, b.nD)[:, :f]
            s["start"] = s["F"][0].clone(), s["F"][1].clone()
    elif case["kind"] == "mlp":
        net = Mlp(s["x"].shape[1], s["t"].shape[1], seed=seed)
        s["net"] = net
        s["X"], rows = net.pad_inputs(torch.from_numpy(s["x"]).to(net.dev))
        s["T"] = torch.zeros((s["X"].shape[0], net.out_p), dtype=torch.float32, device=net.dev)
        s["T"][:rows, :s["t"].shape[1]] = torch.from_numpy(s["t"]).to(net.dev)
    return s


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "als":
        b = state["batch"]
        if case["host"]:
            f = case["rank"]
            b.coef[:f], b.base[:f] = state["start"]
            als.alscpp(b.coef, b.base, b.nbas, f, case["target"], case["sweeps"])
            return b.coef[:f], b.base[:f]
        for part, start in zip(state["F"], state["start"]):
            part.copy_(start)
        als.reduce_batched(state["coef"], state["base"], b.nbas, b.rF, b.rG, b.term_off, case["sweeps"])
        return state["F"]
    if kind == "mlp":
        net = state["net"]
        y = net.forward(state["X"], case["rows"])
        loss = net.backward(state["X"], case["rows"], state["T"])
        net.adam()
        return [y, loss] + [layer[k] for layer in net.layers for k in ("gw", "gb", "w", "b")]
    if kind == "svd":
        return intertwine.reduc_svd(state["base"], state["coef"], [case["nr"], case["nc"]], case["terms"], case["rank"])
    base, coef, hl = state["base"], state["coef"], state["hl"]
    if kind == "cycle":
        return intertwine.intertwine(base, coef, hl.nbas, case["rank"], case["block"], hl, np.zeros(case["block"]),
                                     case["npow"], case["nals"], case["update"], 1, state["shift"],
                                     ranks=state["ranks"])
    if kind == "range":
        return intertwine.spectral_range(base, coef, hl.nbas, case["rank"], hl, case["npow"], case["rounds"])
    if kind == "rayleigh":
        return intertwine.qhq_diag(base, coef, hl.nbas, case["rank"], case["block"], hl)
    if kind == "carry":
        return intertwine.qhq(base, coef, hl.nbas, case["rank"], case["block"], hl)
    return intertwine.diagonalize(base, coef, hl.nbas, case["rank"], case["n"] ** 2, hl, 0)


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------

def work(case):
    """Inputs read once and outputs written once; multiply-adds of the contractions as two operations."""
    kind = case["kind"]
    if kind == "als":
        nd, v, f, g, s = sum(_bases(case)), case["nvec"], case["rank"], case["target"], case["sweeps"]
        flops = v * s * (4.0 * g * nd * f + 2.0 * g * f * case["modes"] + 2.0 * nd * f * f + case["modes"] * f ** 3 / 3.0)
        return {"bytes": 8.0 * v * (nd + 1) * (g + 2 * f), "flops": flops}
    if kind == "mlp":
        m, i, h, o = case["rows"], 64 * (case["n"] + 1), 256, case["n"] * case["rank"]
        w = i * h + h * h + h * o
        return {"bytes": 2.0 * m * i + 4.0 * m * o * 2 + 4.0 * w * 7 + 2.0 * w * 4,
                "flops": 2.0 * m * (2 * w + h * h + h * o)}
    if kind == "svd":
        v, a, b, k = case["nvec"], case["nr"], case["nc"], case["terms"]
        lo, hi = min(a, b), max(a, b)
        return {"bytes": 8.0 * v * (k * (a + b + 1) + case["rank"] * (a + b + 1)),
                "flops": v * (2.0 * k * a * b + 4.0 * hi * lo ** 2 + 8.0 * lo ** 3)}
    if kind == "diag":
        n, r = case["n"], case["rank"]
        b = n * n
        return {"bytes": 8.0 * 2 * b * r * (2 * n + 1), "flops": 9.0 * b ** 3 + b * (2.0 * b * n * n + 12.0 * n ** 3)}
    nb = _bases(case)
    nd, r, d = sum(nb), case["rank"], len(nb)
    if kind == "carry":
        b = case["block"]
        return {"bytes": 8.0 * (b * r * (nd + 1) + b * b),
                "flops": b * r * 2.0 * sum(n * n for n in nb) + b * (b + 1) / 2 * r * r * 2.0 * (nd + d)}
    hl = _operators(case)
    t = hl.nterms
    used = len({(int(o), i % d) for i, o in enumerate(hl.opid)})  # distinct (operator, mode) pairs
    b = {"range": 2}.get(kind) or case["block"]
    grams = used * (2.0 * r * nd * nd / d / d + 2.0 * r * r * nd / d)  # h F and <h F, F> of every pair
    step = 2.0 * t * r * r * d + grams / d + 2.0 * r * r * nd / d + r ** 3 / 3.0  # one mode of one sweep
    if kind == "rayleigh":
        return {"bytes": 8.0 * b * (r * (nd + 1) + 1), "flops": b * (grams + 2.0 * t * r * r * d)}
    if kind == "range":
        return {"bytes": 8.0 * 2 * b * r * (nd + 1), "flops": b * case["rounds"] * (case["npow"] * d * step + grams)}
    p, a = case["npow"], case["nals"]
    flops = b * d * step * (p + (a if case["update"] else 0))
    flops += a * b * b / 2 * r * r * (4.0 * nd + 2.0 * d)  # Gram-Schmidt: overlaps and combinations of earlier vectors
    if case["update"]:
        flops += b * b * r * r * (2.0 * nd + d) + 9.0 * b ** 3 + a * b * b * r * r * (4.0 * nd + d * d)
    return {"bytes": 8.0 * 2 * b * r * (nd + 1), "flops": flops}


# ---------------------------------------------------------------------------
# The same in 64 bits
# ---------------------------------------------------------------------------

def _t(x):
    return torch.as_tensor(np.array(x), dtype=torch.float64, device="cuda" if torch.cuda.is_available() else "cpu")


def _modes(base, nb, block):
    """[block * R, nD] as one [block, R, n] tensor per mode."""
    return [x.reshape(block, -1, int(n)) for x, n in zip(torch.split(_t(base), [int(n) for n in nb], dim=1), nb)]


def _whole(F):
    return torch.cat([f.reshape(-1, f.shape[-1]) for f in F], dim=1)


def _terms(hl):
    """(alpha, per mode the distinct dense operators, per term the operator's place in each mode); place 0: identity."""
    d_of = [[np.eye(int(n))] for n in hl.nbas]
    place, at = [{} for _ in hl.nbas], []
    for i, o in enumerate(hl.opid):
        d = i % len(hl.nbas)
        n = int(hl.nbas[d])
        if o not in place[d]:
            s = int(hl.mptr[o - 1]) - 1
            m = np.zeros((n, n))
            r, c = np.tril_indices(n)
            m[r, c] = m[c, r] = hl.mat[s:s + n * (n + 1) // 2]
            place[d][o] = len(d_of[d])
            d_of[d].append(m)
        at.append(place[d][o])
    return _t(hl.coef), [_t(np.array(m)) for m in d_of], np.array(at).reshape(-1, len(hl.nbas))


def _gram(F):
    return F @ F.transpose(-1, -2)


def _prod(xs):
    out = xs[0].clone()
    for x in xs[1:]:
        out = out * x
    return out


def _norm(F, c):
    return torch.sqrt(torch.abs((c.unsqueeze(-1) * _prod([_gram(f) for f in F]) * c.unsqueeze(-2)).sum((-1, -2))))


def _solve(G, j, b, pen, live):
    """Unit rows of (prod_{d != j} G_d + pen I)^-1 b and their norms; rows beyond a vector's rank stay apart."""
    eye = torch.eye(b.shape[-2], dtype=b.dtype, device=b.device)
    bb = _prod([g for d, g in enumerate(G) if d != j]) + pen[..., None, None] * eye
    if live is not None:
        both = live.unsqueeze(-1) & live.unsqueeze(-2)
        unit = torch.zeros(b.shape[-1], dtype=b.dtype, device=b.device)
        unit[0] = 1.0
        bb, b = torch.where(both, bb, eye.expand_as(bb)), torch.where(live.unsqueeze(-1), b, unit)
    x = torch.linalg.solve(bb, b)
    n = x.norm(dim=-1)
    return x / n.unsqueeze(-1), n if live is None else n * live


def _products(F, c, hl, sweeps, shift, power, live=None):
    """ALS sweeps that fit (H - shift) F: in place, renormalised after each (power), or to the fixed F (not power)."""
    alpha, ops, at = _terms(hl)
    F, Fo, co = [f.clone() for f in F], F, c
    pen = 1e-10 * c.max(dim=-1).values
    applied = lambda d, X: torch.einsum("umn,brn->ubrm", ops[d], X)  # noqa: E731
    Z = [applied(d, f) for d, f in enumerate(Fo)]
    M = [z @ f.transpose(-1, -2) for z, f in zip(Z, F)]
    G = [_gram(f) for f in F]
    rows = [[torch.as_tensor(np.nonzero(at[:, j] == u)[0], device=alpha.device) for u in range(len(ops[j]))]
            for j in range(len(F))]
    where = torch.as_tensor(at, device=alpha.device)
    for _ in range(sweeps):
        for j in range(len(F)):
            W = torch.zeros_like(M[j])
            for u, tt in enumerate(rows[j]):
                for part in torch.split(tt, 16):
                    if len(part):
                        pr = alpha[part].view(-1, 1, 1, 1) * torch.ones_like(M[j][:1])
                        for d in range(len(F)):
                            pr = pr * M[d][where[part, d]] if d != j else pr
                        W[u] += pr.sum(0)
            if power:
                W[0] -= shift.view(-1, 1, 1) * _prod([m[0] for d, m in enumerate(M) if d != j])
            w = W * (c if power else co).unsqueeze(-1)
            b = torch.einsum("ubri,ubrn->bin", w, Z[j])
            F[j], c = _solve(G, j, b, pen, live)
            if power:
                Z[j] = applied(j, F[j])
            M[j] = Z[j] @ F[j].transpose(-1, -2)
            G[j] = _gram(F[j])
            if power:
                c = c / _norm(F, c).unsqueeze(-1)
    return F, c


def _ortho(F, c, sweeps, live=None):
    """The block's vectors in turn fitted to F - sum_k <Q_k, F> Q_k over the earlier ones."""
    F, c = [f.clone() for f in F], c.clone()
    c[0] = c[0] / _norm([f[0] for f in F], c[0])
    for v in range(1, c.shape[0]):
        f, w = [x[v] for x in F], c[v]
        pen = 1e-10 * w.max()
        lv = None if live is None else live[v]
        G = [_gram(x) for x in f]
        P = [q[:v] @ x.transpose(0, 1) for q, x in zip(F, f)]  # [earlier, their terms, terms of the vector]
        for _ in range(sweeps):
            for j in range(len(f)):
                ps = _prod([p for d, p in enumerate(P) if d != j])
                g = -torch.einsum("kr,kri,i->k", c[:v], ps * P[j], w)
                b = (_prod([x for d, x in enumerate(G) if d != j]) * w) @ f[j]
                b = b + torch.einsum("kri,krm->im", ps * (g.unsqueeze(-1) * c[:v]).unsqueeze(-1), F[j][:v])
                f[j], w = _solve(G, j, b, pen, lv)
                G[j], P[j] = _gram(f[j]), F[j][:v] @ f[j].transpose(0, 1)
                w = w / _norm(f, w)
        for x, y in zip(F, f):
            x[v] = y
        c[v] = w
    return F, c


def _inner(F, c, X, w):
    """<X_j, F_i> as [i, j]."""
    rows = []
    for i in range(c.shape[0]):
        p = _prod([x @ f[i].transpose(0, 1) for x, f in zip(X, F)])
        rows.append(torch.einsum("jr,jrs,s->j", w, p, c[i]))
    return torch.stack(rows)


def _geneig(A, S):
    """Ascending eigenpairs of the pencil read from the lower triangles, X^T S X = 1, largest entries positive."""
    low = torch.linalg.cholesky(torch.tril(S) + torch.tril(S, -1).T)
    A = torch.tril(A) + torch.tril(A, -1).T
    y = torch.linalg.solve_triangular(low, A, upper=False)
    e, v = torch.linalg.eigh(torch.linalg.solve_triangular(low, y.T, upper=False))
    x = torch.linalg.solve_triangular(low.T, v, upper=True)
    big = x.gather(0, x.abs().argmax(dim=0, keepdim=True))
    return e, x * torch.sign(big)


def _combine(F, c, U, sweeps):
    """Every vector i fitted to sum_k U(k, i) F_k, from itself."""
    block, R = c.shape
    Q = [f.reshape(block * R, -1) for f in F]
    w = (U.T.unsqueeze(-1) * c.unsqueeze(0)).reshape(block, block * R)
    out, cs, step = [[] for _ in F], [], 10
    for i in range(0, block, step):
        f, n = [x[i:i + step].clone() for x in F], c[i:i + step]
        pen = 1e-10 * n.max(dim=-1).values
        P = [x @ q.T for x, q in zip(f, Q)]
        G = [_gram(x) for x in f]
        for _ in range(sweeps):
            for j in range(len(f)):
                b = (_prod([p for d, p in enumerate(P) if d != j]) * w[i:i + step].unsqueeze(1)) @ Q[j]
                f[j], n = _solve(G, j, b, pen, None)
                P[j], G[j] = f[j] @ Q[j].T, _gram(f[j])
        cs.append(n / _norm(f, n).unsqueeze(-1))
        for o, x in zip(out, f):
            o.append(x)
    return [torch.cat(o) for o in out], torch.cat(cs)


def _quotients(F, c, hl):
    alpha, ops, at = _terms(hl)
    M = [torch.einsum("bim,umn,bjn->ubij", f, o, f) for f, o in zip(F, ops)]
    cc = c.unsqueeze(-1) * c.unsqueeze(-2)
    num = sum(a * (cc * _prod([M[d][u] for d, u in enumerate(row)])).sum((-1, -2)) for a, row in zip(alpha, at))
    return num / (cc * _prod([m[0] for m in M])).sum((-1, -2))


def _exact_als(case, s):
    b, f = s["batch"], case["rank"]
    base = _t(b.base).view(b.nvec, -1, b.nD)
    coef = _t(b.coef).view(b.nvec, -1)
    parts = [int(n) for n in b.nbas]
    F, G = torch.split(base[:, :f], parts, dim=2), torch.split(base[:, f:], parts, dim=2)
    F, c, g = [x / x.norm(dim=-1, keepdim=True) for x in F], coef[:, :f], coef[:, f:]
    pen = 1e-10 * c.max(dim=-1).values
    P, gram = [y @ x.transpose(1, 2) for y, x in zip(G, F)], [_gram(x) for x in F]
    for _ in range(case["sweeps"]):
        for j in range(len(parts)):
            ps = _prod([p for d, p in enumerate(P) if d != j]) * g.unsqueeze(-1)
            F[j], c = _solve(gram, j, ps.transpose(1, 2) @ G[j], pen, None)
            P[j], gram[j] = G[j] @ F[j].transpose(1, 2), _gram(F[j])
    out = c, torch.cat(F, dim=2)
    return tuple(x[0] for x in out) if case["host"] else out


def _exact_mlp(case, s):
    net = Mlp(s["x"].shape[1], s["t"].shape[1], seed=s["seed"])
    p = [[layer[k].double() for layer in net.layers] for k in ("w", "b")]
    rows, rp, outs = case["rows"], -(-case["rows"] // 128) * 128, s["t"].shape[1]
    a = [torch.zeros((rp, net.in_p), dtype=torch.float64, device=net.dev)]
    a[0][:rows, :s["x"].shape[1]] = _t(s["x"])
    for k in range(3):
        z = a[k] @ p[0][k].T + p[1][k]
        z[rows:] = 0.0
        a.append(torch.relu(z) if k < 2 else z)
    d = torch.zeros_like(a[3])
    d[:rows, :outs] = a[3][:rows, :outs] - _t(s["t"])
    got = [a[3], (d ** 2).sum().reshape(1) / (rows * outs)]
    d, grads = 2.0 * d / (rows * outs), []
    for k in (2, 1, 0):
        grads.insert(0, (d.T @ a[k], d.sum(0)))
        d = (d @ p[0][k]) * (a[k] > 0)
    for k, (gw, gb) in enumerate(grads):
        # the first step moves a zero bias by the sign of its gradient alone: no value to hold it to
        got += [gw, gb, p[0][k] - 1e-3 * gw / (gw.abs() + 1e-8), None]
    return got


def exact(case, seed):
    kind, s = case["kind"], _inputs(case, seed)
    if kind == "als":
        return _exact_als(case, s)
    if kind == "mlp":
        return _exact_mlp(case, dict(s, seed=seed))
    if kind == "svd":
        # singular vectors have no sign of their own: the weights and the ranks alone
        b = _t(s["base"]).view(case["nvec"], case["terms"], -1)
        c = _t(s["coef"]).view(case["nvec"], case["terms"], 1)
        sv = torch.linalg.svdvals((c * b[..., :case["nr"]]).transpose(1, 2) @ b[..., case["nr"]:])
        kept = (sv >= 1e-12 * sv[:, :1]).sum(1).clamp(max=case["rank"])
        out = torch.zeros((case["nvec"], case["rank"]), dtype=torch.float64, device=sv.device)
        n = min(case["rank"], sv.shape[1])
        out[:, :n] = sv[:, :n] * (torch.arange(n, device=sv.device) < kept.unsqueeze(1))
        return None, out, kept.to(torch.int32)
    hl, nb = s["hl"], s["hl"].nbas
    if kind == "diag":
        alpha, ops, at = _terms(hl)
        e = torch.linalg.eigvalsh(sum(a * torch.kron(ops[0][u], ops[1][v]) for a, (u, v) in zip(alpha, at)))
        return None, None, e  # the vectors' terms are singular vectors
    block = 2 if kind == "range" else case["block"]
    F, c = _modes(s["base"], nb, block), _t(s["coef"]).view(block, -1)
    if kind == "rayleigh":
        return _quotients(F, c, hl)
    if kind == "carry":
        _, ops, at = _terms(hl)
        return _inner([torch.einsum("mn,brn->brm", o[u], f) for o, u, f in zip(ops, at[0], F)], c, F, c).T
    if kind == "range":
        lo, hi = _quotients(F, c, hl)
        for _ in range(case["rounds"]):
            F, c = _products(F, c, hl, case["npow"], torch.stack([0.5 * (lo + hi), torch.zeros_like(lo)]), True)
            lo, hi = _quotients(F, c, hl)
        pad = 0.001 * (hi - lo)
        return _whole(F), c.reshape(-1), torch.stack([lo - pad, hi + pad])
    live = None
    if s["ranks"] is not None:
        live = torch.arange(case["rank"], device=c.device) < torch.as_tensor(s["ranks"], device=c.device).unsqueeze(1)
        c = c * live
    eig = torch.zeros(block, dtype=torch.float64, device=c.device)
    if case["npow"]:
        F, c = _products(F, c, hl, case["npow"], torch.full((block,), s["shift"], dtype=c.dtype, device=c.device), True,
                         live)
    if case["nals"]:
        F, c = _ortho(F, c, case["nals"], live)
    if case["update"]:
        X, w = _products(F, c, hl, case["nals"], None, False)
        eig, U = _geneig(_inner(X, w, F, c), _inner(F, c, F, c))
        F, c = _combine(F, c, U, case["nals"])
    return _whole(F), c.reshape(-1), eig
