"""Performance cases of the tensor-train solve path, through its public entry points.

Every case is the work of one user call (or one short chain of calls) on
trains that the user's program already holds on the GPU, or, for the batched
solves, on the host, where requests arrive.  The kinds:

* ``dot``: the TTM-by-TT product ``A @ x`` that every residual, matvec and
  time step with an assembled operator starts with; its cores are returned.
* ``truncate``: rounding a sum of two trains (an update, a linear
  combination), ``(p + q).truncate(error)``.
* ``product``: a rounded operator product, ``(A @ x).truncate(error)``.
* ``round_batch``: many pair sums rounded in one launch, ``round_sum_batch``.
* ``tt_svd``: a sampled field compressed into a train.
* ``quantise``: a train turned into its quantised form, ``tt_to_qtt``.
* ``amen``: one linear system, a 2-D Poisson problem in QTT form with a
  right-hand side of a few sine modes, through the drop-in ``amen``.
* ``solve_batch``: many independent systems in one ``amen_persistent`` call,
  QTT Poisson problems or parametric diffusion on ``[0, 1]^d``.

A train is defined only up to the signs and rotations of its bonds, so the
kinds that orthogonalise return the values the train stands for (on the grid,
as the program that wanted the rounded sum or the solution reads them).
"""

from __future__ import annotations

import math

import numpy as np
import torch

import ttnumpy_b200 as tt
from ttnumpy_b200 import problems
from ttnumpy_b200.persistent import amen_persistent
from ttnumpy_b200.rounding import SLOT, PackedTrains, RoundPlan, round_sum_batch

#: AMEn arguments of the serving workload: every solve runs to the tolerance
#: or the sweep cap.  Diffusion solves ask for a digit more than the QTT ones,
#: whose direct local solves end far below the tolerance anyway.
SOLVE = dict(residual_tol=1e-8, symmetric=True, max_sweeps=20, seed=0, stagnation_factor=None)
SOLVE_DIFFUSION = dict(SOLVE, residual_tol=1e-9)


def listed():
    return [
        # residual of a QTT system, 20 cores of mode 2: one tiny product per core, launches count
        {"name": "dot_qtt", "kind": "dot", "op": "poisson", "d": 20, "n": 2, "rank": 8},
        # the same step for a discretised diffusion operator (bond 4) in 12 dimensions, mode 64
        {"name": "dot_diffusion", "kind": "dot", "op": "diffusion", "d": 12, "n": 64, "rank": 32},
        # a small update in QTT form: everything is latency
        {"name": "truncate_qtt", "kind": "truncate", "d": 16, "n": 2, "rank": 5, "error": 1e-8},
        # one pair of the batched rounding workload (mode 4, rank 32 + 32), alone
        {"name": "truncate_pair", "kind": "truncate", "d": 8, "n": 4, "rank": 32, "error": 1e-6},
        # a matvec with the diffusion operator, rounded: bond 96, mode 32
        {"name": "truncate_product", "kind": "product", "d": 4, "n": 32, "rank": 24,
         "error": 1e-8},
        # a handful of pairs: one launch that leaves most of the chip idle
        {"name": "round_few", "kind": "round_batch", "pairs": 12, "d": 10, "n": 2, "rank": 9,
         "error": 1e-8},
        # many pairs of trains of mode 4, rank 32 + 32, rounded to 1e-6
        {"name": "round_many", "kind": "round_batch", "pairs": 512, "d": 8, "n": 4, "rank": 32,
         "error": 1e-6},
        # compressing a sampled three-dimensional field
        {"name": "tt_svd_field", "kind": "tt_svd", "d": 3, "n": 64, "error": 1e-8},
        # a mode-64 train into 18 cores of mode 2
        {"name": "quantise", "kind": "quantise", "d": 3, "n": 64, "rank": 24, "error": 1e-10},
        # one Poisson problem on a 512 x 512 grid, 18 QTT cores
        {"name": "amen_qtt", "kind": "amen", "levels": 9},
        # a batch of QTT Poisson requests of uneven size, one persistent launch
        {"name": "solve_qtt", "kind": "solve_batch", "op": "poisson", "count": 32, "low": 3,
         "high": 8},
        # a batch of parametric diffusion requests, mode 32: iterative local solves
        {"name": "solve_diffusion", "kind": "solve_batch", "op": "diffusion", "count": 8, "d": 4,
         "n": 32},
    ]


def _logint(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["dot", "truncate", "truncate", "product", "round_batch", "round_batch",
                       "tt_svd", "quantise", "amen", "solve_batch"])
    if kind == "dot":
        if rng.random() < 0.5:
            return {"kind": kind, "op": "poisson", "d": 2 * rng.randint(3, 10), "n": 2,
                    "rank": _logint(rng, 2, 40)}
        return {"kind": kind, "op": "diffusion", "d": rng.randint(4, 12),
                "n": rng.choice([16, 24, 32, 49, 64]), "rank": _logint(rng, 3, 32)}
    if kind == "truncate":
        n = rng.choice([2, 3, 4, 5, 8])
        most = int(math.log(1 << 18) / math.log(n))
        return {"kind": kind, "d": rng.randint(4, most), "n": n, "rank": _logint(rng, 3, 32),
                "error": 10.0 ** -rng.uniform(4, 9)}
    if kind == "product":
        return {"kind": kind, "d": rng.randint(3, 4), "n": rng.choice([16, 21, 24, 32]),
                "rank": _logint(rng, 4, 24), "error": 10.0 ** -rng.uniform(6, 9)}
    if kind == "round_batch":
        n = rng.choice([2, 3, 4])
        d = rng.randint(4, {2: 14, 3: 9, 4: 7}[n])
        return {"kind": kind, "pairs": min(_logint(rng, 4, 400), (1 << 24) // n ** d), "d": d,
                "n": n, "rank": rng.randint(4, 32), "error": 10.0 ** -rng.uniform(4, 9)}
    if kind == "tt_svd":
        d, n = rng.choice([(3, 24), (3, 33), (3, 48), (3, 60), (4, 12), (4, 17), (4, 20), (5, 9)])
        return {"kind": kind, "d": d, "n": n, "error": 10.0 ** -rng.uniform(5, 9)}
    if kind == "quantise":
        return {"kind": kind, "d": rng.randint(2, 3), "n": rng.choice([16, 32, 64]),
                "rank": _logint(rng, 3, 24), "error": 10.0 ** -rng.uniform(6, 10)}
    if kind == "amen":
        return {"kind": kind, "levels": rng.randint(3, 9)}
    if rng.random() < 0.6:
        low = rng.randint(3, 5)
        return {"kind": kind, "op": "poisson", "count": _logint(rng, 2, 32), "low": low,
                "high": rng.randint(low, 8)}
    return {"kind": kind, "op": "diffusion", "count": _logint(rng, 2, 24), "d": rng.randint(3, 4),
            "n": rng.choice([12, 15, 16, 24])}


# -- inputs -------------------------------------------------------------------


def _sine_modes(rng, terms=3):
    """A right-hand side of a few sine modes with random amplitudes: the callable the problem
    builder samples, and the (amplitude, i, j) list."""
    modes = [(float(rng.uniform(0.5, 1.5)), int(rng.integers(1, 4)), int(rng.integers(1, 4)))
             for _ in range(terms)]

    def f(x, y):
        return sum(c * np.sin(i * np.pi * x) * np.sin(j * np.pi * y) for c, i, j in modes)

    return f, modes


def _trains(rng, d, n, rank):
    """Uniform [0, 1) cores, the distribution of ``rand``."""
    r = [1] + [rank] * (d - 1) + [1]
    return [rng.random((r[k], n, 1, r[k + 1])) for k in range(d)]


def _levels(case):
    """Grid levels of a batch's requests, spread over the case's range."""
    span = case["high"] - case["low"] + 1
    return [case["low"] + i % span for i in range(case["count"])]


def _operator(case, rng):
    if case["op"] == "poisson":
        return problems.qtt_laplacian_2d(case["d"] // 2, 1.0 / (2 ** (case["d"] // 2) + 1))
    return problems.diffusion_operator(case["d"], case["n"], rng.uniform(-1, 1, case["d"]),
                                       problems.diffusion_scale(case["d"]))


def _field(case, rng):
    """A smooth field on a grid of [0, 1]^d: inverse multiquadrics around random centres and a
    travelling wave."""
    d, n = case["d"], case["n"]
    axes = np.meshgrid(*[np.linspace(0.0, 1.0, n)] * d, indexing="ij", sparse=True)
    f = np.zeros([n] * d)
    for _ in range(3):
        c, w = rng.random(d), rng.uniform(0.1, 0.3)
        f += rng.uniform(0.5, 1.5) / np.sqrt(w ** 2 + sum((a - x) ** 2 for a, x in zip(axes, c)))
    k = rng.uniform(2.0, 8.0, d)
    return f + np.sin(sum(a * b for a, b in zip(axes, k)))


def _host(case, seed):
    """The case's inputs on the host."""
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "dot":
        return _operator(case, rng), _trains(rng, case["d"], case["n"], case["rank"])
    if kind in ("truncate", "round_batch"):
        count = case.get("pairs", 1)
        return tuple([_trains(rng, case["d"], case["n"], case["rank"]) for _ in range(count)]
                     for _ in range(2))
    if kind == "product":
        A = _operator({**case, "op": "diffusion"}, rng)
        return A, _trains(rng, case["d"], case["n"], case["rank"])
    if kind == "tt_svd":
        return _field(case, rng)
    if kind == "quantise":
        return _trains(rng, case["d"], case["n"], case["rank"])
    if kind == "amen":
        return problems.qtt_poisson_2d(case["levels"], _sine_modes(rng)[0])
    if case["op"] == "poisson":
        return [problems.qtt_poisson_2d(size, _sine_modes(rng)[0]) for size in _levels(case)]
    return [problems.parametric_diffusion(case["d"], case["n"], rng.uniform(-1, 1, case["d"]))
            for _ in range(case["count"])]


def prepare(case, seed):
    host = _host(case, seed)
    kind = case["kind"]
    state = {"kind": kind, "error": case.get("error")}
    if kind in ("dot", "product"):
        state["A"], state["x"] = tt.TensorTrain(host[0]), tt.TensorTrain(host[1])
    elif kind == "truncate":
        state["p"], state["q"] = tt.TensorTrain(host[0][0]), tt.TensorTrain(host[1][0])
    elif kind == "round_batch":
        p, q = (PackedTrains.from_numpy(side) for side in host)
        state["p"], state["q"] = p, q
        state["plan"] = RoundPlan(p.count, len(p.modes), p.modes, p.bonds, q.bonds, p.offsets,
                                  q.offsets)
    elif kind == "tt_svd":
        state["field"] = torch.from_numpy(host).to("cuda")
    elif kind == "quantise":
        state["t"] = tt.TensorTrain(host)
    elif kind == "amen":
        state["A"], state["b"] = tt.TensorTrain(host.A), tt.TensorTrain(host.b)
    else:
        # requests as they arrive: host cores, solved in one persistent launch
        args = SOLVE if case["op"] == "poisson" else SOLVE_DIFFUSION
        state["requests"] = [(p.A, p.b, None, dict(args)) for p in host]
    return state


# -- one pass -----------------------------------------------------------------


def _values(res):
    """The values of every rounded train of a batch, as one (pairs, n^d) tensor: the packed cores
    padded to the batch's largest bond and multiplied out."""
    pairs, d, n = res.out.shape[0], len(res.modes), res.modes[0]
    bonds = res.bonds.long()
    top = int(bonds.max())
    dev = res.out.device
    a = torch.arange(top, device=dev).view(1, top, 1, 1)
    i = torch.arange(n, device=dev).view(1, 1, n, 1)
    b = torch.arange(top, device=dev).view(1, 1, 1, top)
    acc = None
    for k in range(d):
        left, right = bonds[:, k].view(-1, 1, 1, 1), bonds[:, k + 1].view(-1, 1, 1, 1)
        ak = a[:, :1] if k == 0 else a
        bk = b[..., :1] if k == d - 1 else b
        inside = ((ak < left) & (bk < right)).expand(pairs, ak.shape[1], n, bk.shape[3])
        at = torch.where(inside, k * SLOT + (ak * n + i) * right + bk, 0)
        core = torch.gather(res.out, 1, at.reshape(pairs, -1))
        core = torch.where(inside.reshape(pairs, -1), core, 0.0).view(pairs, ak.shape[1], -1)
        acc = core if acc is None else torch.bmm(acc, core)
        acc = acc.reshape(pairs, -1, bk.shape[3])
    return acc.view(pairs, -1)


def run(state):
    kind = state["kind"]
    if kind == "dot":
        return (state["A"] @ state["x"]).cores
    if kind == "truncate":
        return (state["p"] + state["q"]).truncate(error=state["error"]).matricize()
    if kind == "product":
        return (state["A"] @ state["x"]).truncate(error=state["error"]).matricize()
    if kind == "round_batch":
        return _values(round_sum_batch(state["p"], state["q"], state["error"], plan=state["plan"]))
    if kind == "tt_svd":
        return tt.tt_svd(state["field"], error=state["error"]).matricize()
    if kind == "quantise":
        return state["t"].tt_to_qtt(mode_size=2, error=state["error"]).matricize()
    if kind == "amen":
        return tt.amen(state["A"], state["b"], **SOLVE).matricize()
    return [r.x.matricize() for r in amen_persistent(state["requests"])]


# -- what a pass cannot do without --------------------------------------------


def _orth_flops(modes, ranks):
    """Householder QR of every unfolding with its Q, then an SVD sweep of the same sizes (its QR
    and its Q; the iteration on the small triangle not counted)."""
    total = 0.0
    for k in range(len(modes) - 1):
        m, c = ranks[k] * modes[k], ranks[k + 1]
        p = min(m, c)
        total += 2 * (4.0 * m * c * p - 4.0 / 3.0 * p ** 3) + 2.0 * p * c * modes[k + 1]
    return total


def _ranks(modes, rank):
    """Bonds of a train of nominal bond ``rank`` after both orthogonalisations."""
    d = len(modes)
    left, right = [1] * (d + 1), [1] * (d + 1)
    for k in range(1, d):
        left[k] = min(rank, left[k - 1] * modes[k - 1])
    for k in range(d - 1, 0, -1):
        right[k] = min(rank, right[k + 1] * modes[k])
    return [min(a, b) for a, b in zip(left, right)]


def _train_size(modes, rank):
    r = [1] + [rank] * (len(modes) - 1) + [1]
    return sum(r[k] * n * r[k + 1] for k, n in enumerate(modes))


def work(case):
    kind = case["kind"]
    if kind == "dot":
        d, n, r = case["d"], case["n"], case["rank"]
        R = 6 if case["op"] == "poisson" else 4
        outs = _train_size([n] * d, R * r)
        ins = _train_size([n] * d, r) + _train_size([n * n] * d, R)
        return {"bytes": 8.0 * (outs + ins), "flops": 2.0 * n * outs}
    if kind in ("truncate", "round_batch"):
        d, n, r = case["d"], case["n"], case["rank"]
        pairs = case.get("pairs", 1)
        return {"bytes": 8.0 * pairs * (2 * _train_size([n] * d, r) + n ** d),
                "flops": pairs * _orth_flops([n] * d, _ranks([n] * d, 2 * r))}
    if kind == "product":
        d, n, r = case["d"], case["n"], case["rank"]
        return {"bytes": 8.0 * (_train_size([n] * d, r) + _train_size([n * n] * d, 4) + n ** d),
                "flops": _orth_flops([n] * d, _ranks([n] * d, 4 * r))}
    if kind == "tt_svd":
        size = float(case["n"] ** case["d"])
        return {"bytes": 16.0 * size, "flops": 4.0 * size * case["n"]}
    if kind == "quantise":
        d, n, r = case["d"], case["n"], case["rank"]
        q = d * int(round(math.log2(n)))
        return {"bytes": 8.0 * (_train_size([n] * d, r) + n ** d),
                "flops": _orth_flops([2] * q, _ranks([2] * q, 2 * r))}
    if kind == "amen":
        return _solve_work("poisson", [case["levels"]], 1)
    if case["op"] == "poisson":
        mid = (case["low"] + case["high"]) // 2
        return _solve_work("poisson", [mid], case["count"])
    return _solve_work("diffusion", [case["d"], case["n"]], case["count"])


def _solve_work(op, size, count):
    """Two sweeps with direct local solves at bond 8 (Poisson), or five with twenty applications
    of the local operator per site at bond 12 (diffusion)."""
    if op == "poisson":
        d = 2 * size[0]
        unknowns = 2 * 8 * 8
        flops = 4.0 * d * (2.0 / 3.0) * unknowns ** 3
        return {"bytes": 8.0 * count * (d * (36 * 4 + 64) + 2.0 ** d), "flops": count * flops}
    d, n = size
    flops = 10.0 * d * 20 * 2.0 * (4 * 12 * n * 12 * (12 + 12) + 15 * n * 12 * 12)
    return {"bytes": 8.0 * count * (16.0 * d * n * n + float(n) ** d), "flops": count * flops}


# -- exact values -------------------------------------------------------------


def _full(cores):
    t = cores[0].reshape(-1, cores[0].shape[-1])
    for c in cores[1:]:
        t = (t @ c.reshape(c.shape[0], -1)).reshape(-1, c.shape[-1])
    return t.reshape(-1)


def _bond(s, delta):
    s = np.where(s <= np.finfo(float).eps * s.size * s[0], 0.0, s)
    tail = np.cumsum((s ** 2)[::-1])[::-1]
    return max(1, int(np.count_nonzero(tail > delta * delta)))


def _rounded(cores, error):
    """The textbook rounding: a left-to-right QR sweep, then a right-to-left SVD sweep that drops
    a tail of at most ``error * norm / sqrt(d - 1)`` per bond."""
    cores = [c.reshape(c.shape[0], -1, c.shape[-1]) for c in cores]
    d = len(cores)
    for k in range(d - 1):
        a, n, b = cores[k].shape
        q, r = np.linalg.qr(cores[k].reshape(a * n, b))
        cores[k] = q.reshape(a, n, -1)
        cores[k + 1] = np.einsum("ij,jnk->ink", r, cores[k + 1])
    delta = error / math.sqrt(d - 1) * np.linalg.norm(cores[-1])
    for k in range(d - 1, 0, -1):
        a, n, b = cores[k].shape
        u, s, vh = np.linalg.svd(cores[k].reshape(a, n * b), full_matrices=False)
        nb = _bond(s, delta)
        cores[k] = vh[:nb].reshape(nb, n, b)
        cores[k - 1] = cores[k - 1] @ (u[:, :nb] * s[:nb])
    return cores


def _sum(p, q):
    out = []
    for k, (a, b) in enumerate(zip(p, q)):
        if k == 0:
            out.append(np.concatenate([a, b], axis=3))
        elif k == len(p) - 1:
            out.append(np.concatenate([a, b], axis=0))
        else:
            c = np.zeros((a.shape[0] + b.shape[0], a.shape[1], 1, a.shape[3] + b.shape[3]))
            c[: a.shape[0], :, :, : a.shape[3]] = a
            c[a.shape[0]:, :, :, a.shape[3]:] = b
            out.append(c)
    return out


def _product(A, x):
    out = []
    for a, c in zip(A, x):
        y = np.einsum("aijb,xjky->axikby", a, c, optimize=True)
        out.append(y.reshape(a.shape[0] * c.shape[0], a.shape[1], c.shape[2], -1))
    return out


def exact(case, seed):
    host = _host(case, seed)
    kind = case["kind"]
    if kind == "dot":
        return _product(*host)
    if kind == "truncate":
        return _full(_rounded(_sum(host[0][0], host[1][0]), case["error"]))
    if kind == "product":
        return _full(_rounded(_product(*host), case["error"]))
    if kind == "round_batch":
        if case["pairs"] * case["d"] * case["rank"] ** 2 > 1 << 22:
            return None  # over twenty seconds of host factorisations
        return np.stack([_full(_rounded(_sum(p, q), case["error"])) for p, q in zip(*host)])
    if kind == "tt_svd":
        d, n = case["d"], case["n"]
        delta = case["error"] / math.sqrt(d - 1) * np.linalg.norm(host)
        cores, rest, bond = [], host.reshape(-1), 1
        for _ in range(d - 1):
            mat = rest.reshape(bond * n, -1)
            u, s, _ = np.linalg.svd(mat, full_matrices=False)
            nb = _bond(s, delta)
            cores.append(u[:, :nb].reshape(bond, n, nb))
            rest, bond = u[:, :nb].T @ mat, nb
        return _full(cores + [rest.reshape(bond, n, 1)])
    if kind == "quantise":
        return _full(host)  # to the requested error, far above rounding
    if kind == "amen":
        return _poisson_solution(case["levels"], np.random.default_rng(seed))
    if case["op"] == "poisson":
        rng = np.random.default_rng(seed)
        return [_poisson_solution(size, rng) for size in _levels(case)]
    return None  # a system of n^d unknowns with a varying coefficient, per request


def _poisson_solution(levels, rng):
    """The discrete solution: sine modes are eigenvectors of the five-point Laplacian."""
    modes = _sine_modes(rng)[1]
    size = 2 ** levels
    h = 1.0 / (size + 1)
    nodes = (np.arange(size) + 1) * h
    out = np.zeros((size, size))
    for c, i, j in modes:
        lam = 4 / h ** 2 * (math.sin(i * math.pi * h / 2) ** 2 + math.sin(j * math.pi * h / 2) ** 2)
        out += c / lam * np.outer(np.sin(j * math.pi * nodes), np.sin(i * math.pi * nodes))
    return out.reshape(-1)
