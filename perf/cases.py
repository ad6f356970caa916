"""Performance cases of the simulator: what its users run, through the public
entry points of for-qaoa_b200/forqaoa.py and for-qaoa_b200/sharded.py.

Five kinds of work, each over the range of sizes its users have:
  forward    Context.qaoa_forward: the state vector and <C> of one circuit
  gradient   Context.energy_grad: one step of an optimiser loop
  serve      Server: a burst of optimiser steps from many sessions
  reference  Context.reference_schedule (per-launcher kernels in FOR-QAOA's
             own order), then the state in logical order and <C>, as a
             drop-in user and the driver's --dump have it
  sharded    sharded.forward with every shard on this GPU (the per-rank
             passes of a multi-GPU run, the exchange as device copies)
Graphs are the ones of the tests and the benchmark: complete with integer
weights 1..10, G(n, 1/2) with integer or signed integer weights, G(n, 1/2)
with FP64 weights in [0, 1), and random 3-regular with FP64 weights; angles
are uniform, gamma in [0, pi), beta in [0, pi/2).
"""
import os
import sys

import numpy as np
import torch

HERE = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(HERE, "for-qaoa_b200"))

import forqaoa  # noqa: E402
import sharded  # noqa: E402

GRAPHS = ("complete_int", "gnp_int", "gnp_signed", "gnp_fp", "regular3_fp")


def listed():
    return [
        # The smallest calls: a teaching-size circuit, latency only.
        dict(name="forward_n9_p2", kind="forward", n=9, p=2, graph="gnp_int"),
        # The accuracy configuration: K_20, p=5, whole state and <C>.
        dict(name="forward_n20_p5", kind="forward", n=20, p=5, graph="complete_int"),
        # An odd size with FP64 weights, the state about half of L2.
        dict(name="forward_n23_p4_fp", kind="forward", n=23, p=4, graph="gnp_fp"),
        # Sparse FP64 graph on a state well beyond L2 (3-regular, p=3).
        dict(name="forward_n28_p3_reg3", kind="forward", n=28, p=3, graph="regular3_fp"),
        # The headline circuit: K_30, p=5, a 16 GiB state.
        dict(name="forward_n30_p5", kind="forward", n=30, p=5, graph="complete_int"),
        # Optimiser steps, one at a time: small enough for one SM ...
        dict(name="gradient_n12_p4", kind="gradient", n=12, p=4, graph="gnp_int"),
        # ... a few SMs ...
        dict(name="gradient_n15_p6", kind="gradient", n=15, p=6, graph="gnp_fp"),
        # ... an odd size whose two vectors stay in L2 ...
        dict(name="gradient_n19_p6", kind="gradient", n=19, p=6, graph="gnp_int"),
        # ... and the gradient configuration, K_26, p=10, two 1 GiB vectors.
        dict(name="gradient_n26_p10", kind="gradient", n=26, p=10, graph="complete_int"),
        # A burst of requests at a server, mixed sizes and depths.
        dict(name="serve_96_n10_20", kind="serve", requests=96, lo=10, hi=20, graph="gnp_int"),
        # The drop-in path with the driver's chunk size, state beyond L2.
        dict(name="reference_n26_c12_p2", kind="reference", n=26, c=12, p=2, graph="complete_int"),
        # Two shards of a 27-qubit state.
        dict(name="sharded_n27_d1_p2", kind="sharded", n=27, d=1, p=2, graph="complete_int"),
    ]


def draw(rng):
    kind = rng.choice(("forward", "forward", "gradient", "gradient", "serve", "reference",
                       "sharded"))
    graph = rng.choice(GRAPHS)
    if kind == "forward":
        return dict(kind=kind, n=rng.randint(4, 29), p=rng.randint(1, 8), graph=graph)
    if kind == "gradient":
        return dict(kind=kind, n=rng.randint(4, 26), p=rng.randint(1, 10), graph=graph)
    if kind == "serve":
        lo = rng.randint(8, 16)
        return dict(kind=kind, requests=rng.randint(16, 160), lo=lo,
                    hi=rng.randint(lo + 1, 21), graph="gnp_int")
    if kind == "reference":
        return dict(kind=kind, n=rng.randint(14, 27), c=rng.randint(10, 13), p=rng.randint(1, 3),
                    graph=graph)
    return dict(kind=kind, n=rng.randint(18, 28), d=rng.randint(1, 3), p=rng.randint(1, 3),
                graph=graph)


# ---- inputs -----------------------------------------------------------------
def make_graph(name, n, rng):
    """Upper-triangular N x N weights (0 = no edge)."""
    if name == "regular3_fp":
        m = n + n % 2  # 3-regular needs an even number; an odd n drops one vertex's edges
        while True:
            pairs = rng.permutation(np.repeat(np.arange(m), 3)).reshape(-1, 2)
            edges = {tuple(sorted(e)) for e in pairs.tolist()}
            if len(edges) == len(pairs) and all(a != b for a, b in edges):
                break
        w = np.zeros((n, n))
        for a, b in sorted(edges):
            if b < n:
                w[a, b] = rng.random()
        return w
    if name == "complete_int":
        w = rng.integers(1, 11, (n, n)).astype(np.float64)
    elif name == "gnp_int":
        w = rng.integers(1, 11, (n, n)) * (rng.random((n, n)) < 0.5)
    elif name == "gnp_signed":
        w = rng.integers(-10, 11, (n, n)) * (rng.random((n, n)) < 0.5)
    else:
        w = rng.random((n, n)) * (rng.random((n, n)) < 0.5)
    return np.triu(w, 1).astype(np.float64)


def angles(p, rng):
    return rng.uniform(0, np.pi, p), rng.uniform(0, np.pi / 2, p)


def circuit(case, seed):
    rng = np.random.default_rng([seed, 30])
    g = make_graph(case["graph"], case["n"], rng)
    return (g,) + angles(case["p"], rng)


def requests(case, seed):
    """Sizes and depths belong to the case; graphs and angles to the seed."""
    sizes = np.random.default_rng([case["requests"], case["lo"], case["hi"]])
    rng = np.random.default_rng([seed, 31])
    out = []
    for _ in range(case["requests"]):
        n, p = int(sizes.integers(case["lo"], case["hi"] + 1)), int(sizes.integers(1, 9))
        out.append((make_graph(case["graph"], n, rng),) + angles(p, rng))
    return out


class Amplitudes:
    """A device state as a tensor without a copy; it frees the state, and the
    context when it owns one, with the last tensor on it."""

    def __init__(self, ctx, n):
        self.ctx, self.state = ctx, ctx.state(n)
        self.__cuda_array_interface__ = {"shape": (1 << n,), "typestr": "<c16", "version": 3,
                                         "data": (self.state.ptr.value, False)}

    def tensor(self):
        return torch.as_tensor(self, device="cuda")

    def __del__(self):
        self.state.free()


class Handle:
    """Closes a context or server when the last user of it is gone."""

    def __init__(self, obj):
        self.obj = obj

    def __getattr__(self, name):
        return getattr(self.obj, name)

    def __del__(self):
        self.obj.close()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "serve":
        return dict(kind=kind, server=Handle(forqaoa.Server(0, hbm_budget_bytes=20e9, lanes=4)),
                    requests=requests(case, seed))
    graph, gammas, betas = circuit(case, seed)
    n = case["n"]
    s = dict(kind=kind, n=n, graph=graph, gammas=gammas, betas=betas)
    if kind == "sharded":
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            s["stream"], s["d"] = stream, case["d"]
            s["ctx"] = Handle(forqaoa.Context(0, stream.cuda_stream))
            s["shards"] = [sharded.ShardOps(s["ctx"], n, case["d"], r, "cuda")
                           for r in range(1 << case["d"])]
        return s
    ctx = s["ctx"] = Handle(forqaoa.Context(0))
    if kind == "forward":
        s["psi"] = Amplitudes(ctx, n)
    elif kind == "gradient":
        big = n > forqaoa.SMALL_MAX_QUBITS  # smaller instances need no buffers
        s["psi"] = Amplitudes(ctx, n) if big else None
        s["costate"] = Amplitudes(ctx, n) if big else None
    else:
        s["c"] = case["c"]
        s["psi"], s["logical"] = Amplitudes(ctx, n), Amplitudes(ctx, n)
        s["labels"] = forqaoa.reference_label_map(n, case["c"], case["p"])
    return s


def run(s):
    kind = s["kind"]
    if kind == "forward":
        e = s["ctx"].qaoa_forward(s["psi"].state, s["graph"], s["gammas"], s["betas"])
        return {"energy": e, "psi": s["psi"].tensor()}
    if kind == "gradient":
        sv, cs = (x.state if x else None for x in (s["psi"], s["costate"]))
        e, gg, gb = s["ctx"].energy_grad(s["n"], s["graph"], s["gammas"], s["betas"], sv, cs)
        return {"energy": e, "grad_gamma": gg, "grad_beta": gb}
    if kind == "serve":
        tickets = [s["server"].submit(i, g, ga, be)
                   for i, (g, ga, be) in enumerate(s["requests"])]
        done = s["server"].wait(tickets)
        res = [done[t] for t in tickets]
        return {"energy": np.array([r.energy for r in res]),
                "grad_gamma": np.concatenate([r.grad_gamma for r in res]),
                "grad_beta": np.concatenate([r.grad_beta for r in res])}
    if kind == "reference":
        ctx = s["ctx"]
        g = ctx.reference_schedule(s["psi"].state, s["graph"], s["c"], s["gammas"], s["betas"])
        ctx.permute_qubits(s["psi"].state, s["logical"].state, s["labels"])
        e = ctx.expectation(s["logical"].state, s["graph"])
        return {"energy": e, "psi": s["logical"].tensor(), "graph": g}
    with torch.cuda.stream(s["stream"]):
        _, g = sharded.forward(s["shards"], sharded.local_exchange, s["n"], s["d"], s["graph"],
                               s["gammas"], s["betas"])
        e = sum(x.expectation(g) for x in s["shards"])
    return {"energy": e, "graph": g, "psi": [x.buf for x in s["shards"]]}


# ---- work ---------------------------------------------------------------------
def circuit_flops(n, p):
    """A rotation is two multiply-adds per amplitude and qubit, a phase one
    complex product per amplitude."""
    return p * 2.0 ** n * (4 * n + 6)


def gradient_flops(n, p):
    """Forward, and both vectors back with the two inner products."""
    return 3 * circuit_flops(n, p) + p * 2.0 ** n * (4 * n + 6)


def work(case):
    kind = case["kind"]
    if kind == "serve":
        rs = requests(case, 0)
        return {"bytes": float(sum(8 * (g.size + 4 * len(ga) + 1) for g, ga, _ in rs)),
                "flops": float(sum(gradient_flops(g.shape[0], len(ga)) for g, ga, _ in rs))}
    n, p = case["n"], case["p"]
    small = 8.0 * (n * n + 2 * p + 1)
    if kind == "gradient":
        return {"bytes": small + 16.0 * p, "flops": gradient_flops(n, p)}
    return {"bytes": small + 16.0 * 2.0 ** n, "flops": circuit_flops(n, p)}


# ---- the same in plain torch, 64 bits ---------------------------------------------
def cut_values(w):
    """C(z) of every z, bit by bit: qubit n adds w_in (z_i xor z_n)."""
    c = torch.zeros(1, dtype=torch.float64, device="cuda")
    for n in range(w.shape[0]):
        lin = torch.zeros(1, dtype=torch.float64, device="cuda")
        for i in range(n):
            lin = torch.cat([lin, lin + w[i, n]])
        c = torch.cat([c + lin, c + (w[:n, n].sum() - lin)])
    return c


def rotate(psi, q, beta):
    v = psi.view(-1, 2, 1 << q)
    c, s = float(np.cos(beta / 2)), float(np.sin(beta / 2))
    a, b = v[:, 0].clone(), v[:, 1].clone()
    v[:, 0].mul_(c).add_(b, alpha=-1j * s)
    v[:, 1].mul_(c).add_(a, alpha=-1j * s)


def phase(psi, cut, total, gamma):
    step = 1 << 26
    for i in range(0, psi.numel(), step):
        x = (2 * cut[i:i + step] - total) * gamma / 2
        psi[i:i + step].mul_(torch.polar(torch.ones_like(x), x))


def exact_state(g, gammas, betas, cut):
    n = g.shape[0]
    psi = torch.full((1 << n,), 2.0 ** (-n / 2), dtype=torch.complex128, device="cuda")
    for gamma, beta in zip(gammas, betas):
        phase(psi, cut, g.sum(), gamma)
        for q in range(n):
            rotate(psi, q, beta)
    return psi


def mean_cut(psi, cut):
    step = 1 << 26
    return sum(float(((x := torch.view_as_real(psi[i:i + step])).square().sum(1)
                      * cut[i:i + step]).sum()) for i in range(0, psi.numel(), step))


def inner_im(a, b):
    return float((a.real * b.imag - a.imag * b.real).sum())


def exact_gradient(g, gammas, betas):
    n, p, total = g.shape[0], len(gammas), g.sum()
    cut = cut_values(g)
    psi = exact_state(g, gammas, betas, cut)
    energy = mean_cut(psi, cut)
    lam = psi * cut
    gg, gb = np.zeros(p), np.zeros(p)
    for k in reversed(range(p)):
        for q in range(n):
            v = psi.view(-1, 2, 1 << q).flip(1).reshape(-1)
            gb[k] += inner_im(lam, v)
        for q in range(n):
            rotate(psi, q, -betas[k])
            rotate(lam, q, -betas[k])
        gg[k] = -inner_im(lam * (2 * cut - total), psi)
        phase(psi, cut, total, -gammas[k])
        phase(lam, cut, total, -gammas[k])
    return energy, gg, gb


def swapped(g, labels, out, into, k):
    """Labels and graph after qubit blocks [out, out+k) and [into, into+k)
    trade places."""
    n = len(labels)
    pos = np.arange(n)
    pos[out:out + k], pos[into:into + k] = np.arange(into, into + k), np.arange(out, out + k)
    full = g + g.T
    return np.triu(full[np.ix_(pos, pos)], 1), labels[pos]


def exact(case, seed):
    kind = case["kind"]
    if kind == "serve":
        res = [exact_gradient(*r) for r in requests(case, seed)]
        return {"energy": np.array([r[0] for r in res]),
                "grad_gamma": np.concatenate([r[1] for r in res]),
                "grad_beta": np.concatenate([r[2] for r in res])}
    graph, gammas, betas = circuit(case, seed)
    if kind == "gradient":
        return dict(zip(("energy", "grad_gamma", "grad_beta"),
                        exact_gradient(graph, gammas, betas)))
    n, cut = case["n"], cut_values(graph)
    psi = exact_state(graph, gammas, betas, cut)
    out = {"energy": mean_cut(psi, cut), "psi": psi}
    if kind == "forward":
        return out
    g, labels = graph, np.arange(n)
    for _ in range(case["p"]):
        if kind == "sharded":
            d = case["d"]
            g, labels = swapped(g, labels, n - 2 * d, n - d, d)
        else:
            sizes = [min(case["c"], n - i) for i in range(0, n, case["c"])]
            for i in range(1, len(sizes)):
                g, labels = swapped(g, labels, 0, sum(sizes[:i]), sizes[i])
    out["graph"] = g
    if kind == "sharded":  # physical order: position b holds logical qubit labels[b]
        dims = [n - 1 - int(q) for q in reversed(labels)]
        psi = psi.view([2] * n).permute(dims).reshape(-1)
        out["psi"] = list(psi.chunk(1 << case["d"]))
    return out
