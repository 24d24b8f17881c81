"""The workloads that the performance figures of this framework are measured on.

Every case is one public call as a user's program makes it: a network right-hand side, a
derivative of it, a time integration, a batch of steady states, a training step of the
learned warm start.  Sizes are those of the reference's benchmark networks, of this
repository's benchmarks and tests, or lie between them.

``listed()`` names the cases, ``draw(rng)`` gives another one of the same ranges,
``prepare(case, seed)`` builds what a program has in hand before the call (graph, network
handle, states and parameters made from the seed), ``run(state)`` makes the call, ``work``
counts the bytes and operations it cannot do without, and ``exact`` computes the same
outputs in 64 bits with plain torch.
"""
import functools
import math
import random
import sys
from pathlib import Path

import numpy as np
import torch

_ROOT = Path(__file__).resolve().parent.parent
if str(_ROOT / "networkdynamics.jl_gb300") not in sys.path:
    sys.path.insert(0, str(_ROOT / "networkdynamics.jl_gb300"))

import nd_gb300 as nd  # noqa: E402
from nd_gb300.ensemble import Ensemble  # noqa: E402
from nd_gb300.solve import solve_tsit5  # noqa: E402

_DEV = "cuda"
_BITS = {"f64": torch.float64, "f32": torch.float32, "f32x2": "f32x2"}


def listed():
    return [
        # the smallest networks a user integrates: one RHS is launch latency
        {"name": "rhs_kuramoto_ws1k_f64", "what": "rhs", "model": "kuramoto", "graph": "ws", "n": 1000, "k": 10,
         "beta": 0.1, "dtype": "f64"},
        # the swing equations on a mid-size scale-free grid (hubs of ~1000 lines, a sine per line)
        {"name": "rhs_swing_ba100k_f64", "what": "rhs", "model": "swing", "graph": "ba", "n": 100_000, "k": 2,
         "beta": 0.0, "dtype": "f64"},
        # diffusion on a large scale-free network: the headline workload's model, memory-bound
        {"name": "rhs_diffusion_ba2m_f64", "what": "rhs", "model": "diffusion", "graph": "ba", "n": 2_000_000, "k": 4,
         "beta": 0.0, "dtype": "f64"},
        # the same model in the other precision
        {"name": "rhs_diffusion_ba1m_f32", "what": "rhs", "model": "diffusion", "graph": "ba", "n": 1_000_000, "k": 4,
         "beta": 0.0, "dtype": "f32"},
        # the reference's diffusion_ode_edge benchmark: edges with states on a dense ring
        {"name": "rhs_ode_edges_ws3k_f64", "what": "ode_edges", "n": 3000, "k": 1500, "dtype": "f64"},
        # the reference's powergrid benchmark: PQ buses, generators and pi-lines
        {"name": "rhs_powergrid_100k_f64", "what": "powergrid", "n": 100_000, "k": 2, "beta": 0.8, "dtype": "f64"},
        # Jacobian-vector product, as a matrix-free implicit solver asks for it
        {"name": "jvp_swing_ba500k_f64", "what": "jvp", "n": 500_000, "k": 2, "dtype": "f64"},
        # the assembled sparse Jacobian, as a stiff solver or a stability analysis asks for it
        {"name": "jacobian_swing_ba100k_f64", "what": "jacobian", "n": 100_000, "k": 2, "dtype": "f64"},
        # one network integrated by adaptive Tsit5
        {"name": "tsit5_swing_ba100k_f64", "what": "tsit5", "n": 100_000, "k": 2, "t_end": 2.0, "dtype": "f64"},
        # basin stability: many instances of different sizes integrated side by side
        {"name": "ensemble_swing_rgg1024_f64", "what": "ensemble", "instances": 1024, "lo": 50, "hi": 2000,
         "t_end": 2.0, "graph_seed": 10, "dtype": "f64"},
        # steady states of one grid under many loads (training data of the warm start)
        {"name": "fixpoint_ba2k_x1000", "what": "fixpoint", "instances": 1000, "n": 2000, "k": 2},
        # one training step of the warm start's message-passing network (forward, backward, Adam)
        {"name": "mpnn_train_ba2k_b64", "what": "mpnn", "n": 2000, "k": 2, "batch": 64, "layers": 4},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["rhs", "rhs", "rhs", "ode_edges", "powergrid", "jvp", "jacobian", "tsit5", "ensemble",
                       "fixpoint", "mpnn"])
    dtype = rng.choice(["f64", "f64", "f32"])
    if what == "rhs":
        model = rng.choice(["diffusion", "kuramoto", "swing"])
        graph = rng.choice(["ba", "ba", "ws", "dense"])
        if graph == "ba":
            return {"what": what, "model": model, "graph": graph, "n": _log_int(rng, 1000, 1_500_000),
                    "k": rng.randint(2, 5), "beta": 0.0, "dtype": dtype}
        if graph == "ws":
            return {"what": what, "model": model, "graph": graph, "n": _log_int(rng, 300, 300_000),
                    "k": 2 * rng.randint(1, 10), "beta": round(rng.uniform(0.0, 0.8), 2), "dtype": dtype}
        n = _log_int(rng, 300, 3000)
        return {"what": what, "model": model, "graph": "ws", "n": n, "k": n // 4 * 2, "beta": 0.0, "dtype": dtype}
    if what == "ode_edges":
        n = _log_int(rng, 300, 3000)
        return {"what": what, "n": n, "k": rng.choice([10, n // 4 * 2]), "dtype": dtype}
    if what == "powergrid":
        return {"what": what, "n": _log_int(rng, 1000, 150_000), "k": 2 * rng.randint(1, 2),
                "beta": round(rng.uniform(0.2, 0.8), 2), "dtype": dtype}
    if what == "jvp":
        return {"what": what, "n": _log_int(rng, 2000, 500_000), "k": rng.randint(2, 4), "dtype": dtype}
    if what == "jacobian":
        return {"what": what, "n": _log_int(rng, 1000, 150_000), "k": rng.randint(2, 4), "dtype": dtype}
    if what == "tsit5":
        return {"what": what, "n": _log_int(rng, 1000, 100_000), "k": rng.randint(2, 3),
                "t_end": round(rng.uniform(0.5, 2.0), 2), "dtype": "f64"}
    if what == "ensemble":
        return {"what": what, "instances": _log_int(rng, 16, 1024), "lo": 50, "hi": _log_int(rng, 100, 2000),
                "t_end": round(rng.uniform(0.5, 2.0), 2), "graph_seed": rng.randint(1, 10**6),
                "dtype": rng.choice(["f64", "f32", "f32x2"])}
    if what == "fixpoint":
        return {"what": what, "instances": _log_int(rng, 16, 1000), "n": _log_int(rng, 100, 2000),
                "k": rng.randint(2, 3)}
    return {"what": what, "n": _log_int(rng, 100, 2000), "k": rng.randint(2, 3), "batch": _log_int(rng, 4, 64),
            "layers": rng.randint(2, 4)}


# ---- graphs (of the case, not of the seed: a program keeps its graph) -------------------------

@functools.lru_cache(maxsize=4)
def _graph(kind, n, k, beta):
    return nd.barabasi_albert(n, k, seed=1) if kind == "ba" else nd.watts_strogatz(n, k, beta, seed=1)


@functools.lru_cache(maxsize=2)
def _instances(count, lo, hi, seed):
    """Random geometric graphs of mean degree 6, sizes U[lo, hi]."""
    r = random.Random(seed)
    sizes = [r.randint(lo, hi) for _ in range(count)]
    return [nd.random_geometric(n, math.sqrt(6.0 / (math.pi * n)), seed=seed + 10 + i) for i, n in enumerate(sizes)]


def _case_graph(case):
    return _graph(case.get("graph", "ba"), case["n"], case["k"], case.get("beta", 0.0))


def _ends(g):
    return torch.from_numpy(g.src).to(_DEV), torch.from_numpy(g.dst).to(_DEV)


# ---- inputs -----------------------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device=_DEV).manual_seed(int(seed))


def _uniform(gen, lo, hi, *size):
    return torch.rand(*size, generator=gen, device=_DEV, dtype=torch.float64) * (hi - lo) + lo


def _normal(gen, *size):
    return torch.randn(*size, generator=gen, device=_DEV, dtype=torch.float64)


def _injections(gen, *size):
    """Balanced power injections: generators and loads in turn, each row summing to zero."""
    p = _uniform(gen, 0.5, 1.5, *size)
    p[..., 1::2] *= -1.0
    return p - p.mean(-1, keepdim=True)


def _swing_vertex_params(pm):
    out = torch.empty(*pm.shape, 3, device=_DEV, dtype=torch.float64)
    out[..., 0], out[..., 1], out[..., 2] = 1.0, 0.1, pm
    return out.flatten(-2)


def _model_inputs(case, seed):
    """u and p (64 bits) of a homogeneous network."""
    g, gen, model = _case_graph(case), _gen(seed), case.get("model", "swing")
    if model == "diffusion":
        return _normal(gen, g.nv), _uniform(gen, 0.0, 1.0, g.ne)
    if model == "kuramoto":
        return _uniform(gen, -math.pi, math.pi, g.nv), torch.cat([_normal(gen, g.nv), _uniform(gen, 0.5, 1.5, g.ne)])
    u = torch.empty(g.nv, 2, device=_DEV, dtype=torch.float64)
    near = case["what"] == "tsit5"  # from near the synchronous state, as a stability study starts
    u[:, 0] = 0.3 * _normal(gen, g.nv) if near else _uniform(gen, -math.pi, math.pi, g.nv)
    u[:, 1] = 0.0 if near else _normal(gen, g.nv)
    return u.flatten(), torch.cat([_swing_vertex_params(_injections(gen, g.nv)), _uniform(gen, 5.0, 10.0, g.ne)])


def _ode_inputs(case, seed):
    g, gen = _graph("ws", case["n"], case["k"], 0.0), _gen(seed)
    return g, _normal(gen, g.nv + 2 * g.ne)


def _grid_kinds(n):
    """0: PQ bus, 1: generator; half of each, shuffled."""
    return np.random.default_rng(1).permutation(np.arange(n) % 2)


def _grid_layout(n):
    """First state and first parameter of every vertex: batches in order of first appearance."""
    kinds = _grid_kinds(n)
    order = [int(kinds[0]), 1 - int(kinds[0])]
    s, q = np.empty(n, np.int64), np.empty(n, np.int64)
    s0 = q0 = 0
    for b in order:
        at = np.flatnonzero(kinds == b)
        s[at], q[at] = s0 + np.arange(at.size) * (2, 4)[b], q0 + np.arange(at.size) * (2, 11)[b]
        s0, q0 = s0 + at.size * (2, 4)[b], q0 + at.size * (2, 11)[b]
    return kinds, s, q, s0, q0


def _grid_inputs(case, seed):
    """Per-unit states and machine / line data."""
    g, gen = _graph("ws", case["n"], case["k"], case["beta"]), _gen(seed)
    kinds, _, q, dim, npar = _grid_layout(g.nv)
    p = torch.empty(npar + 4 * g.ne, device=_DEV, dtype=torch.float64)
    qt = torch.from_numpy(q).to(_DEV)
    pq, mach = (torch.from_numpy(np.flatnonzero(kinds == b)).to(_DEV) for b in (0, 1))
    for k in range(2):
        p[qt[pq] + k] = _uniform(gen, -1.0, 1.0, pq.numel())
    data = (5.0, None, 0.1, 2 * math.pi * 50, 1.0, 7.0, 0.5, 0.3, 0.6, 1.8, 1.7)
    for k, x in enumerate(data):
        p[qt[mach] + k] = _uniform(gen, -1.0, 1.0, mach.numel()) if x is None \
            else x * _uniform(gen, 0.9, 1.1, mach.numel())
    line = p[npar:].view(g.ne, 4)
    for k, x in enumerate((1e-3, 0.05, 1e-5, 1e-5)):
        line[:, k] = x * _uniform(gen, 0.8, 1.2, g.ne)
    return g, 1.0 + 0.1 * _normal(gen, dim), p


def _ensemble_inputs(case, seed):
    """Packed u and p: phases near the synchronous state, one vertex of each instance knocked off it."""
    gs, gen = _instances(case["instances"], case["lo"], case["hi"], case["graph_seed"]), _gen(seed)
    nv, ne = sum(g.nv for g in gs), sum(g.ne for g in gs)
    u = torch.zeros(nv, 2, device=_DEV, dtype=torch.float64)
    u[:, 0] = 0.2 * _normal(gen, nv)
    first = np.concatenate([[0], np.cumsum([g.nv for g in gs])[:-1]])
    hit = torch.from_numpy(first).to(_DEV)
    u[hit, 0] += _uniform(gen, -math.pi, math.pi, len(gs))
    u[hit, 1] += _uniform(gen, -10.0, 10.0, len(gs))
    pm, k = _uniform(gen, 0.5, 1.5, nv), _uniform(gen, 5.0, 10.0, ne)
    parts, v, e = [], 0, 0
    for g in gs:
        x = pm[v:v + g.nv].clone()
        x[1::2] *= -1.0
        parts += [_swing_vertex_params(x - x.mean()), k[e:e + g.ne]]
        v, e = v + g.nv, e + g.ne
    return gs, u.flatten(), torch.cat(parts)


def _fixpoint_inputs(case, seed):
    g, gen, b = _case_graph(case), _gen(seed), case["instances"]
    return g, _injections(gen, b, g.nv), _uniform(gen, 5.0, 10.0, b, g.ne)


def _mpnn_inputs(case, seed):
    g, gen, b = _case_graph(case), _gen(seed), case["batch"]
    nparams = 192 + case["layers"] * 8256 + 65
    P, K = _injections(gen, b, g.nv).float(), _uniform(gen, 5.0, 10.0, b, g.ne).float()
    T, w = (0.3 * _normal(gen, b, g.nv)).float(), _uniform(gen, -0.15, 0.15, nparams).float()
    return g, P, K, T, w


# ---- the calls ----------------------------------------------------------------------------------

_MODELS = {"diffusion": (nd.diffusion_vertex, nd.diffusion_edge), "kuramoto": (nd.kuramoto_first, nd.kuramoto_edge),
           "swing": (nd.kuramoto_second, nd.static_line)}


def prepare(case, seed):
    what = case["what"]
    st = {"what": what, "case": case}
    if what in ("rhs", "jvp", "jacobian", "tsit5"):
        dt = _BITS[case["dtype"]]
        vm, em = _MODELS[case.get("model", "swing")]
        st["nw"] = nd.adapt(nd.Network(_case_graph(case), vm(), em()), dt)
        u, p = _model_inputs(case, seed)
        st["u"], st["p"] = u.to(dt), p.to(dt)
        if what == "jvp":
            st["v"] = _normal(_gen(seed + 1), u.numel()).to(dt)
        if what == "jacobian":
            nd.jacobian_pattern(st["nw"])  # the prototype, built once per network
        st["out"] = torch.empty_like(st["u"])
    elif what == "ode_edges":
        g, u = _ode_inputs(case, seed)
        st["nw"] = nd.adapt(nd.Network(g, nd.diffusion_vertex(), nd.diffusion_dedge()), _BITS[case["dtype"]])
        st["u"], st["p"] = u.to(_BITS[case["dtype"]]), None
        st["out"] = torch.empty_like(st["u"])
    elif what == "powergrid":
        g, u, p = _grid_inputs(case, seed)
        vm = (nd.pqnode(), nd.generator())
        st["nw"] = nd.adapt(nd.Network(g, [vm[k] for k in _grid_kinds(g.nv)], nd.piline()), _BITS[case["dtype"]])
        st["u"], st["p"] = u.to(_BITS[case["dtype"]]), p.to(_BITS[case["dtype"]])
        st["out"] = torch.empty_like(st["u"])
    elif what == "ensemble":
        gs, u, p = _ensemble_inputs(case, seed)
        st["ens"] = Ensemble(gs, nd.kuramoto_second(), nd.static_line(), _BITS[case["dtype"]])
        st["u"], st["p"] = u, p.to(st["ens"].torch_dtype)
    elif what == "fixpoint":
        g, P, K = _fixpoint_inputs(case, seed)
        st["ens"] = Ensemble([g] * case["instances"], nd.kuramoto_second(), nd.static_line(), torch.float64)
        st["p"] = torch.cat([_swing_vertex_params(P), K], 1).flatten()
        st["u"] = torch.zeros(2 * P.numel(), device=_DEV, dtype=torch.float64)
    else:
        g, st["P"], st["K"], st["T"], w = _mpnn_inputs(case, seed)
        st["model"] = nd.MPNN(g, layers=case["layers"])
        st["model"].set_params(w)
    return st


def run(st):
    what = st["what"]
    if what in ("rhs", "ode_edges", "powergrid"):
        st["nw"](st["out"], st["u"], st["p"], 0.0)
        return st["out"]
    if what == "jvp":
        nd.jvp(st["nw"], st["out"], st["u"], st["p"], st["v"])
        return st["out"]
    if what == "jacobian":
        J = nd.jacobian(st["nw"], st["u"], st["p"])
        return [J.crow_indices(), J.col_indices(), J.values()]
    if what == "tsit5":
        return solve_tsit5(st["nw"], st["u"], st["p"], (0.0, st["case"]["t_end"]), reltol=1e-6, abstol=1e-8)[0]
    if what == "ensemble":
        r = st["ens"].solve_tsit5(st["u"], st["p"], (0.0, st["case"]["t_end"]), reltol=1e-6, abstol=1e-6)
        return [r.u, r.status]
    if what == "fixpoint":
        r = st["ens"].fixpoint(st["u"], st["p"], tol=1e-10)
        return [r.u, r.status]
    loss = st["model"].loss_grad(st["P"], st["K"], st["T"])
    grads = st["model"].get_grads()
    st["model"].adam_step(lr=1e-3)
    return [loss, grads]


# ---- what a pass cannot do without ---------------------------------------------------------------

def work(case):
    """Bytes: states, parameters and results once, and the edge list once (8 bytes an edge).
    Operations: a sine or cosine as 20, a division as 10, of each edge and vertex once per
    evaluation of the right-hand side."""
    what = case["what"]
    s = 4 if case.get("dtype") == "f32" else 8
    if what == "ode_edges":
        e = case["n"] * (case["k"] // 2)
        return {"bytes": s * 2 * (case["n"] + 2 * e) + 8 * e, "flops": 27 * e}
    if what == "powergrid":
        n, e = case["n"], case["n"] * (case["k"] // 2)
        return {"bytes": s * (2 * 3 * n + 6.5 * n + 4 * e) + 8 * e, "flops": 60 * e + 80 * n}
    if what == "ensemble":
        n = case["instances"] * (case["lo"] + case["hi"]) / 2
        e, steps = 3 * n, 16 * case["t_end"]
        return {"bytes": 8 * 4 * n + s * (3 * n + e) + 8 * e, "flops": steps * (6 * (24 * e + 16 * n) + 110 * n)}
    n = case["n"]
    e = n * (case["k"] // 2) if case.get("graph") == "ws" else n * case["k"]
    if what == "fixpoint":
        b = case["instances"]
        return {"bytes": b * 8 * (2 * n + 3 * n + e + 2 * n) + 8 * e, "flops": b * (4 * 24 * e + 250 * (4 * e + 10 * n))}
    if what == "mpnn":
        b, layers = case["batch"], case["layers"]
        dense = 3 * layers * 2 * b * n * 128 * 64
        return {"bytes": 4 * b * (2 * n + e) + 8 * e, "flops": dense + 2 * layers * b * 4 * e * 64}
    dim, par, f = {"diffusion": (n, e, 4 * e), "kuramoto": (n, n + e, 24 * e + n),
                   "swing": (2 * n, 3 * n + e, 24 * e + 14 * n)}[case.get("model", "swing")]
    if what == "jacobian":
        nnz = 3 * n + 2 * e
        return {"bytes": s * (dim + par + nnz) + 8 * (nnz + dim) + 8 * e, "flops": f}
    if what == "jvp":
        return {"bytes": s * (3 * dim + par) + 8 * e, "flops": f + 4 * e}
    if what == "tsit5":
        steps = 100 * case["t_end"]
        return {"bytes": s * (2 * dim + par) + 8 * e, "flops": steps * (6 * f + 55 * dim)}
    return {"bytes": s * (2 * dim + par) + 8 * e, "flops": f}


# ---- the same outputs in 64 bits with plain torch --------------------------------------------------

def _as_given(x, case):
    """What the call sees: inputs rounded to its precision."""
    return x.float().double() if case.get("dtype") == "f32" else x


def _edge_sum(n, src, dst, y):
    """Every vertex's sum of its edges' flows: +y at the destination, -y at the source."""
    return torch.zeros(n, device=_DEV, dtype=torch.float64).index_add_(0, dst, y).index_add_(0, src, -y)


def _swing_rhs(u, src, dst, M, D, Pm, K):
    th, w = u[0::2], u[1::2]
    acc = _edge_sum(th.numel(), src, dst, K * torch.sin(th[src] - th[dst]))
    return torch.stack([w, (Pm - D * w + acc) / M], 1).flatten()


def _rk4(f, u, t_end, h):
    steps = max(1, int(math.ceil(t_end / h)))
    h = t_end / steps
    for _ in range(steps):
        k1 = f(u)
        k2 = f(u + 0.5 * h * k1)
        k3 = f(u + 0.5 * h * k2)
        k4 = f(u + h * k3)
        u = u + (h / 6.0) * (k1 + 2.0 * k2 + 2.0 * k3 + k4)
    return u


def _exact_swing(case, seed):
    g = _case_graph(case)
    src, dst = _ends(g)
    u, p = (_as_given(x, case) for x in _model_inputs(case, seed))
    q = p[:3 * g.nv].view(-1, 3)
    return g, src, dst, u, q[:, 0], q[:, 1], q[:, 2], p[3 * g.nv:]


def _exact_rhs(case, seed):
    g = _case_graph(case)
    src, dst = _ends(g)
    if case["model"] == "swing":
        g, src, dst, u, M, D, Pm, K = _exact_swing(case, seed)
        return _swing_rhs(u, src, dst, M, D, Pm, K)
    u, p = (_as_given(x, case) for x in _model_inputs(case, seed))
    if case["model"] == "diffusion":
        return _edge_sum(g.nv, src, dst, p * (u[src] - u[dst]))
    return p[:g.nv] + _edge_sum(g.nv, src, dst, p[g.nv:] * torch.sin(u[src] - u[dst]))


def _exact_ode_edges(case, seed):
    g, u = _ode_inputs(case, seed)
    src, dst = _ends(g)
    u = _as_given(u, case)
    v, e = u[:g.nv], u[g.nv:].view(-1, 2)
    flow = torch.sin(v[src] - v[dst])
    dv = torch.zeros(g.nv, device=_DEV, dtype=torch.float64).index_add_(0, dst, e[:, 0]).index_add_(0, src, e[:, 1])
    return torch.cat([dv, torch.stack([100.0 * (flow - e[:, 0]), 100.0 * (-flow - e[:, 1])], 1).flatten()])


def _exact_powergrid(case, seed):
    g, u, p = _grid_inputs(case, seed)
    u, p = _as_given(u, case), _as_given(p, case)
    src, dst = _ends(g)
    kinds, s, q, dim, npar = _grid_layout(g.nv)
    s, q = torch.from_numpy(s).to(_DEV), torch.from_numpy(q).to(_DEV)
    omega = 2 * math.pi * 50 if case["dtype"] != "f32" else float(np.float32(2 * math.pi * 50))
    V = torch.complex(u[s], u[s + 1])
    L, R, C1, C2 = p[npar:].view(-1, 4).T
    main = (V[src] - V[dst]) / torch.complex(R, omega * L)
    ysrc, ydst = main + V[src] * (1j * omega * C1), -(main - V[dst] * (1j * omega * C2))
    cur = torch.zeros(g.nv, device=_DEV, dtype=torch.complex128).index_add_(0, src, ysrc).index_add_(0, dst, ydst)
    du = torch.empty(dim, device=_DEV, dtype=torch.float64)
    at = torch.from_numpy(np.flatnonzero(kinds == 0)).to(_DEV)
    x = torch.complex(p[q[at]], p[q[at] + 1]) / cur[at].conj()
    du[s[at]], du[s[at] + 1] = x.real, x.imag
    at = torch.from_numpy(np.flatnonzero(kinds == 1)).to(_DEV)
    H, P, D, Om, Ef, Td, Tq, Xqd, Xdd, Xd, Xq = (p[q[at] + k] for k in range(11))
    i, uc, th, w = cur[at], V[at], u[s[at] + 2], u[s[at] + 3]
    turn = torch.polar(torch.ones_like(th), -th)
    ic, ec = 1j * i * turn, 1j * uc * turn
    ded = (-ec.real + (Xq - Xqd) * ic.imag) / Tq
    deq = (-ec.imag - (Xd - Xdd) * ic.real + Ef) / Td
    d = torch.complex(deq, -ded) * turn.conj() + uc * 1j * w
    du[s[at]], du[s[at] + 1], du[s[at] + 2] = d.real, d.imag, w
    du[s[at] + 3] = (P - D * w - (uc * i.conj()).real - (Xqd - Xdd) * ic.real * ic.imag) * (Om / (2 * H))
    return du


def _exact_jvp(case, seed):
    g, src, dst, u, M, D, _, K = _exact_swing(case, seed)
    v = _as_given(_normal(_gen(seed + 1), u.numel()), case)
    th, x = u[0::2], v[0::2]
    acc = _edge_sum(g.nv, src, dst, K * torch.cos(th[src] - th[dst]) * (x[src] - x[dst]))
    return torch.stack([v[1::2], (acc - D * v[1::2]) / M], 1).flatten()


def _exact_jacobian(case, seed):
    g, src, dst, u, M, D, _, K = _exact_swing(case, seed)
    c = K * torch.cos(u[0::2][src] - u[0::2][dst])
    v = torch.arange(g.nv, device=_DEV)
    row = torch.cat([2 * v, 2 * v + 1, 2 * dst + 1, 2 * src + 1, 2 * dst + 1, 2 * src + 1])
    col = torch.cat([2 * v + 1, 2 * v + 1, 2 * src, 2 * dst, 2 * dst, 2 * src])
    val = torch.cat([torch.ones_like(M), -D / M, c / M[dst], c / M[src], -c / M[dst], -c / M[src]])
    at, where = torch.unique(row * (2 * g.nv) + col, return_inverse=True)
    values = torch.zeros(at.numel(), device=_DEV, dtype=torch.float64).index_add_(0, where, val)
    crow = torch.zeros(2 * g.nv + 1, device=_DEV, dtype=torch.int64)
    crow[1:] = torch.cumsum(torch.bincount(at // (2 * g.nv), minlength=2 * g.nv), 0)
    return [crow, at % (2 * g.nv), values]


def _exact_tsit5(case, seed):
    g, src, dst, u, M, D, Pm, K = _exact_swing(case, seed)
    # hubs of degree d oscillate at up to sqrt(2 d K): the step follows the fastest one
    h = 0.1 / math.sqrt(20.0 * float(g.degree().max()))
    return _rk4(lambda x: _swing_rhs(x, src, dst, M, D, Pm, K), u, case["t_end"], h)


def _exact_ensemble(case, seed):
    gs, u, p = _ensemble_inputs(case, seed)
    p = _as_given(p, case)
    src, dst, par, line, v, q = [], [], [], [], 0, 0
    for g in gs:
        src.append(g.src + v)
        dst.append(g.dst + v)
        par.append(p[q:q + 3 * g.nv])
        line.append(p[q + 3 * g.nv:q + 3 * g.nv + g.ne])
        v, q = v + g.nv, q + 3 * g.nv + g.ne
    src, dst = (torch.from_numpy(np.concatenate(x)).to(_DEV) for x in (src, dst))
    M, D, Pm = torch.cat(par).view(-1, 3).T
    K = torch.cat(line)
    return [_rk4(lambda x: _swing_rhs(x, src, dst, M, D, Pm, K), u, case["t_end"], 0.004), None]


def _exact_fixpoint(case, seed):
    """Newton on the power balance; each linear system by conjugate gradients."""
    g, P, K = _fixpoint_inputs(case, seed)
    src, dst = _ends(g)

    def flows(y):
        return torch.zeros_like(P).index_add_(1, dst, y).index_add_(1, src, -y)

    th = torch.zeros_like(P)
    for _ in range(6):
        diff = th[:, src] - th[:, dst]
        r = P + flows(K * torch.sin(diff))
        r = r - r.mean(1, keepdim=True)
        if float(r.abs().max()) < 1e-13:
            break
        wgt = K * torch.cos(diff)
        x, d, rr = torch.zeros_like(r), r.clone(), (r * r).sum(1, keepdim=True)
        stop = 1e-18 * rr + 1e-30
        for it in range(4 * g.nv):
            q = -flows(wgt * (d[:, src] - d[:, dst]))
            on = rr > stop  # instances that are done keep their solution
            a = torch.where(on, rr / (d * q).sum(1, keepdim=True), torch.zeros_like(rr))
            x, r = x + a * d, r - a * q
            rn = (r * r).sum(1, keepdim=True)
            d = torch.where(on, r + rn / rr * d, d)
            rr = rn
            if it % 16 == 0 and not bool(on.any()):
                break
        th = th + x - x.mean(1, keepdim=True)
    return [torch.stack([th, torch.zeros_like(th)], 2).flatten(), None]


def _exact_mpnn(case, seed):
    g, P, K, T, w = _mpnn_inputs(case, seed)
    src, dst = _ends(g)
    b, n, layers = case["batch"], g.nv, case["layers"]
    P, K, T, w = P.double(), K.double() / 10.0, T.double(), w.double().requires_grad_()
    s = torch.zeros_like(P).index_add_(1, dst, K).index_add_(1, src, K)
    inv = torch.where(s > 0, 1.0 / s, torch.zeros_like(s)).unsqueeze(2)

    def mat(at, rows, cols):
        return w[at:at + rows * cols].view(rows, cols)

    h = torch.tanh(torch.stack([P, torch.log1p(s)], 2) @ mat(0, 64, 2).T + w[128:192])
    for k in range(layers):
        at = 192 + 8256 * k
        m = torch.zeros_like(h).index_add(1, dst, K.unsqueeze(2) * h[:, src])
        m = inv * m.index_add(1, src, K.unsqueeze(2) * h[:, dst])
        h = h + torch.tanh(h @ mat(at, 64, 64).T + m @ mat(at + 4096, 64, 64).T + w[at + 8192:at + 8256])
    y = h @ w[-65:-1] + w[-1]
    e = (y - y.mean(1, keepdim=True)) - (T - T.mean(1, keepdim=True))
    loss = (e * e).sum() / (b * n)
    loss.backward()
    return [loss.detach(), w.grad]


_EXACT = {"rhs": _exact_rhs, "ode_edges": _exact_ode_edges, "powergrid": _exact_powergrid, "jvp": _exact_jvp,
          "jacobian": _exact_jacobian, "tsit5": _exact_tsit5, "ensemble": _exact_ensemble,
          "fixpoint": _exact_fixpoint, "mpnn": _exact_mpnn}


def exact(case, seed):
    return _EXACT[case["what"]](case, seed)
