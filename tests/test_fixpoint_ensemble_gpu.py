"""Batched steady states of swing networks whose solve must not be taken for a solution, and of
networks that are not connected."""
import numpy as np
import pytest

import nd_gb300 as nd
from nd_gb300 import _capi as capi
from nd_gb300 import warmstart as W
from nd_gb300.ensemble import Ensemble
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def swing_flat(P, K):
    return np.concatenate([np.stack([np.ones(P.size), np.full(P.size, 0.1), P], 1).ravel(), K])


def solve(graphs, ps, **options):
    import torch
    ens = Ensemble(graphs, nd.kuramoto_second(), nd.static_line(), torch.float64)
    r = ens.fixpoint(torch.zeros(ens.dim, dtype=torch.float64, device="cuda"),
                     torch.from_numpy(np.concatenate(ps)).cuda(), **options)
    return ens, r.u.cpu().numpy(), r.status.cpu().numpy(), r.resid.cpu().numpy()


@pytest.mark.parametrize("nv", [4, 300])  # fewer rows than a warp; more than a block has threads
@pytest.mark.parametrize("where", ["every vertex", "first vertex", "last vertex", "a line"])
def test_nan_is_not_converged(cuda, nv, where):
    """A NaN in one row's power balance or in all of them is reported, with a NaN residual, and
    the other instances of the batch are solved."""
    g = nd.cycle_graph(nv)
    P = np.where(np.arange(nv) % 2 == 0, 1.0, -1.0)
    good = swing_flat(P, np.full(g.ne, 6.0))
    Q, K = P.copy(), np.full(g.ne, 6.0)
    if where == "a line":
        K[nv // 2] = np.nan
    else:
        Q[{"every vertex": slice(None), "first vertex": 0, "last vertex": -1}[where]] = np.nan
    ens, u, status, resid = solve([g, g, g], [good, swing_flat(Q, K), good])
    assert status.tolist() == [capi.ND_OK, capi.ND_ERR_NOT_CONVERGED, capi.ND_OK]
    assert np.isnan(resid[1]) and np.all(resid[[0, 2]] <= 1e-10)
    for i in (0, 2):
        th = u[ens.u_slice(i)][0::2]
        np.testing.assert_allclose(np.abs(np.diff(th)), np.arcsin(1 / 12), atol=1e-11)


def disjoint(parts):
    """The parts side by side, as one graph."""
    src, dst, nv = [], [], 0
    for g in parts:
        src.append(g.src + nv)
        dst.append(g.dst + nv)
        nv += g.nv
    return nd.Graph(nv, np.concatenate(src).astype(np.int64), np.concatenate(dst).astype(np.int64))


def balanced(g, P):
    """P without its mean over every connected component."""
    import scipy.sparse as sp
    from scipy.sparse.csgraph import connected_components
    n, label = connected_components(sp.coo_matrix((np.ones(g.ne), (g.src, g.dst)), shape=(g.nv, g.nv)), directed=False)
    return P - (np.bincount(label, weights=P, minlength=n) / np.bincount(label, minlength=n))[label], label


def assert_sound(g, u, p, status, resid):
    """OK only with a finite state whose right-hand side, by the oracle, is as small as reported
    (1e-10, and 1e-13 of the rows' terms for the two sums)."""
    if status != capi.ND_OK:
        return
    on = O.OracleNetwork.from_graph(g, O.V_SWING, O.E_KURAMOTO)
    assert np.all(np.isfinite(u)) and resid <= 1e-10
    assert np.all(np.abs(on.rhs(u, p)) <= 1e-10 + 1e-13 * on.abs_terms(u, p))


def test_overloaded_network_in_twelve_components(cuda):
    """A random geometric graph of twelve components (six of them single vertices) whose lines cannot
    carry its injections: Newton does not converge and must not say so."""
    g = nd.random_geometric(1516, float(np.sqrt(6.0 / (np.pi * 1516))), seed=552)
    P, K = W.swing_instances(g, 1, 116380)
    p = W.swing_flat_params(g, P, K)
    ens, u, status, resid = solve([g], [p], max_newton=12, max_cg=4000)
    assert status[0] == capi.ND_ERR_MAXITERS
    assert np.all(np.isfinite(u)) and np.isfinite(resid[0])


@pytest.mark.parametrize("load", [0.02, 0.3, 1.0])  # carried by all, by some and by few of the graphs
def test_random_geometric_components(cuda, load):
    """Sixty-four sparse geometric graphs of 20 to 700 vertices, nearly all with isolated vertices and
    pairs: what is reported as solved is a steady state, and at the light load all are."""
    graphs, ps = [], []
    for i, nv in enumerate(np.random.default_rng(3).integers(20, 700, 64)):
        g = nd.random_geometric(int(nv), float(np.sqrt(5.0 / (np.pi * nv))), seed=900 + i)
        P, K = W.swing_instances(g, 1, 77 + i)
        graphs.append(g)
        ps.append(W.swing_flat_params(g, load * P, K))
    ens, u, status, resid = solve(graphs, ps, max_newton=15)
    for i, g in enumerate(graphs):
        assert_sound(g, u[ens.u_slice(i)], ps[i], status[i], resid[i])
    assert np.all(np.isfinite(u))
    if load < 0.1:
        assert np.all(status == capi.ND_OK)


@pytest.mark.parametrize("sizes", [
    (1,), (1, 1, 1), (40, 1), (500, 32, 33, 1, 2, 31), (300, 300, 300), (600,) + 300 * (1,)])
def test_components_of_every_size(cuda, sizes):
    """Parts a block, a warp and a thread each take: every part's phases are those of the part solved
    alone (the phase shift of each part stays that of the start)."""
    rng = np.random.default_rng(sum(sizes))
    parts = [nd.barabasi_albert(n, 2, seed=n) if n > 2 else nd.simple_graph(n, [(0, 1)][:n - 1]) for n in sizes]
    P = [balanced(g, rng.uniform(-1, 1, g.nv))[0] for g in parts]
    K = [rng.uniform(5, 10, g.ne) for g in parts]
    g = disjoint(parts)
    p = swing_flat(np.concatenate(P), np.concatenate(K))
    both = [g] + parts
    ens, u, status, resid = solve(both, [p] + [swing_flat(a, b) for a, b in zip(P, K)])
    assert np.all(status == capi.ND_OK) and np.all(resid <= 1e-10)
    whole = u[ens.u_slice(0)][0::2]
    alone = np.concatenate([u[ens.u_slice(1 + k)][0::2] for k in range(len(parts))])
    # residuals of 1e-10 a row, over the smallest eigenvalue of a part's weighted Laplacian (above 1
    # here): 1e-10 sqrt(600) for either solve
    np.testing.assert_allclose(whole, alone, atol=5e-9)


@pytest.mark.parametrize("island", ["balanced", "unbalanced"])
def test_lines_of_weight_zero(cuda, island):
    """Two halves joined by lines of weight 0 only: solved where each half is balanced; not, and
    finite, where they are not."""
    a, b = nd.barabasi_albert(400, 2, seed=5), nd.barabasi_albert(300, 2, seed=6)
    two = disjoint([a, b])
    bridge = np.arange(8, dtype=np.int64)
    src, dst = np.concatenate([two.src, bridge]), np.concatenate([two.dst, 400 + bridge])
    order = np.lexsort((dst, src))
    g = nd.Graph(700, np.ascontiguousarray(src[order]), np.ascontiguousarray(dst[order]))
    rng = np.random.default_rng(8)
    K = np.concatenate([rng.uniform(5, 10, two.ne), np.zeros(8)])[order]
    P, _ = balanced(two, rng.uniform(-1, 1, 700))
    if island == "unbalanced":
        P[:400] += 0.01
        P[400:] -= 0.01 * 400 / 300
    p = swing_flat(P, K)
    ens, u, status, resid = solve([g], [p], max_newton=12)
    assert np.all(np.isfinite(u))
    assert_sound(g, u, p, status[0], resid[0])
    assert status[0] == (capi.ND_OK if island == "balanced" else capi.ND_ERR_MAXITERS)
