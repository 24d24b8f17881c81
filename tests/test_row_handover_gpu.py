"""The row kernels that start beside the last blocks of their edge kernel: rows of every length
around their batch of terms, and calls one behind the other, each reading its own edges."""
import numpy as np
import pytest

import nd_gb300 as nd
from nd_gb300.solve import solve_tsit5
from oracle import oracle as O

from ndtest import gpu_rhs

pytestmark = pytest.mark.gpu


def hub_graph(degrees, nv):
    k = len(degrees)
    e = sorted((h, k + i) for h, d in enumerate(degrees) for i in range(d))
    arr = np.array(e, dtype=np.int64)
    return nd.Graph(nv, np.ascontiguousarray(arr[:, 0]), np.ascontiguousarray(arr[:, 1]))


@pytest.mark.parametrize("nv", [63, 64, 65, 129])  # around the blocks of 64 rows and lines
def test_powergrid_rows(cuda, nv):
    """Rows of 0 to 17 lines; lines without resistance, without reactance and without either (both
    branches of the complex division, its zero numerators, and infinities).  No sine: the
    oracle's bits."""
    import torch
    g = hub_graph([0, 1, 2, 3, 4, 5, 7, 8, 9, 12, 13, 16, 17], nv)
    net = nd.Network(g, [nd.pqnode()] * nv, nd.piline())
    on = O.OracleNetwork.from_batches(g.nv, g.src, g.dst, [m.kind for m in net.vertex_batches], net.vertex_batch,
                                      [(O.E_PILINE, O.C_FIDUCIAL)], net.edge_batch)
    rng = np.random.default_rng(nv)
    u, p = rng.normal(size=net.dim), rng.uniform(0.5, 1.5, size=net.pdim)
    line = p[net.pdim - 4 * g.ne:].reshape(-1, 4)
    line[0::5, 1] = 0.0
    line[1::5, 0] = 0.0
    line[7, :2] = 0.0
    u[2 * g.dst[3]:2 * g.dst[3] + 2] = u[2 * g.src[3]:2 * g.src[3] + 2]
    np.testing.assert_array_equal(gpu_rhs(nd.adapt(net, torch.float64), u, p, cuda, np.float64), on.rhs(u, p))


@pytest.mark.parametrize("kind", ["powergrid", "mixed", "two-phase", "dense"])
@pytest.mark.parametrize("dtype", ["float64", "float32"])
def test_calls_in_a_row(cuda, kind, dtype):
    """Twelve calls on twelve states without a synchronisation between them, plain and replayed
    from a captured graph, have the bits of calls made one at a time."""
    import torch
    dt = getattr(torch, dtype)
    if kind == "powergrid":
        g = nd.watts_strogatz(3000, 4, 0.5, seed=1)
        net = nd.Network(g, [nd.pqnode() if i % 3 else nd.generator() for i in range(g.nv)], nd.piline())
    elif kind == "mixed":
        g = nd.watts_strogatz(3000, 6, 0.5, seed=2)
        net = nd.Network(g, [nd.kuramoto_first() if i % 2 else nd.kuramoto_second() for i in range(g.nv)],
                         nd.kuramoto_edge() if hasattr(nd, "kuramoto_edge") else nd.static_line())
    elif kind == "two-phase":
        net = nd.Network(nd.watts_strogatz(220_000, 20, 0.3, seed=3), nd.kuramoto_second(), nd.static_line())
    else:
        net = nd.Network(nd.watts_strogatz(2200, 1100, 0.0, seed=4), nd.diffusion_vertex(), nd.diffusion_edge())
    net = nd.adapt(net, dt)
    gen = torch.Generator(device=cuda).manual_seed(5)
    u = torch.randn(12, net.dim, dtype=dt, device=cuda, generator=gen)
    p = torch.rand(net.pdim, dtype=dt, device=cuda, generator=gen) + 0.5
    ref, got = torch.empty_like(u), torch.zeros_like(u)
    for i in range(12):
        net(ref[i], u[i], p, 0.0)
        torch.cuda.synchronize()
    for i in range(12):
        net(got[i], u[i], p, 0.0)
    torch.cuda.synchronize()
    assert torch.equal(got, ref)
    graph = torch.cuda.CUDAGraph()
    got.zero_()
    with torch.cuda.graph(graph):
        for i in range(12):
            net(got[i], u[i], p, 0.0)
    for _ in range(3):
        got.zero_()
        graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(got, ref)


@pytest.mark.parametrize("n,k", [(2000, 998), (2000, 1000), (1600, 1250)])  # 998,000 edges and from 1e6 on
def test_f32_long_rows_of_mixed_vertices(cuda, n, k):
    """FP32 rows of about k terms, started beside the edge phase or after it: within 4e-6 of the FP64
    oracle's term scale (24 eps of a compensated sum), and twelve calls in a row have the bits of
    calls made one at a time."""
    import torch
    g = nd.watts_strogatz(n, k, 0.3, seed=7)
    net = nd.Network(g, [nd.kuramoto_first() if i % 2 else nd.kuramoto_second() for i in range(n)], nd.kuramoto_edge())
    on = O.OracleNetwork.from_batches(g.nv, g.src, g.dst, [m.kind for m in net.vertex_batches], net.vertex_batch,
                                      [(O.E_KURAMOTO, O.C_ANTISYMMETRIC)], net.edge_batch)
    rng = np.random.default_rng(k)
    us = rng.normal(size=(12, net.dim)).astype(np.float32)
    p = rng.uniform(0.5, 1.5, size=net.pdim).astype(np.float32)
    nw = nd.adapt(net, torch.float32)
    ref = np.stack([gpu_rhs(nw, u, p, cuda, np.float32) for u in us])
    for u, r in zip(us[:2], ref):
        e = on.rhs(u.astype(np.float64), p.astype(np.float64))
        # |terms| <= K <= 1.5 each; the swing rows' division by M >= 0.5
        assert np.all(np.abs(r - e) <= 4e-6 * 2.0 * (1.5 * g.degree().max() + 5.0))
    src, pt = torch.from_numpy(us).to(cuda), torch.from_numpy(p).to(cuda)
    got = torch.empty_like(src)
    for i in range(12):
        nw(got[i], src[i], pt, 0.0)
    np.testing.assert_array_equal(got.cpu().numpy(), ref)


@pytest.mark.parametrize("vertices", ["generators", "swing and kuramoto"])
@pytest.mark.parametrize("nv", [1, 64, 65, 5000])
def test_network_without_edges(cuda, vertices, nv):
    """Rows of a network without edges come behind whatever wrote their states: calls that each
    follow the kernel writing theirs have the bits of calls made one at a time, which are the
    oracle's (sines: 1e-13 of the term scale), and Tsit5 runs through."""
    import torch
    g = nd.simple_graph(nv, [])
    if vertices == "generators":
        net = nd.Network(g, [nd.generator()] * nv, nd.piline())
    else:
        net = nd.Network(g, [nd.kuramoto_second() if i % 2 else nd.kuramoto_first() for i in range(nv)], nd.static_line())
    on = O.OracleNetwork.from_batches(g.nv, g.src, g.dst, [m.kind for m in net.vertex_batches], net.vertex_batch, [], [])
    rng = np.random.default_rng(nv)
    us, p = rng.normal(size=(16, net.dim)), rng.uniform(0.5, 1.5, size=net.pdim)
    nw = nd.adapt(net, torch.float64)
    ref = np.stack([gpu_rhs(nw, u, p, cuda, np.float64) for u in us])
    for u, r in zip(us, ref):
        e = on.rhs(u, p)
        assert np.all(np.abs(r - e) <= 1e-13 * (10.0 + np.abs(e)))
    src, pt = torch.from_numpy(us).to(cuda), torch.from_numpy(p).to(cuda)
    u, got = torch.full((net.dim,), float("nan"), dtype=torch.float64, device=cuda), torch.empty_like(src)
    for i in range(16):
        torch.mul(src[i], 1.0, out=u)
        nw(got[i], u, pt, 0.0)
    np.testing.assert_array_equal(got.cpu().numpy(), ref)
    uT, _ = solve_tsit5(nw, torch.from_numpy(0.1 * us[0]).to(cuda), pt, (0.0, 0.5), reltol=1e-8, abstol=1e-10)
    assert torch.isfinite(uT).all()


@pytest.mark.parametrize("degrees", [tuple(range(18, 36)), (3, 4, 5, 9, 10, 11, 15, 16, 17, 64, 700)])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_powergrid_hubs(cuda, degrees, dtype):
    """Rows of more lines than the first batch and the next ones hold: the oracle's bits in FP64; FP32
    as near to it as its own rounding of sums of `n` currents and one division allows."""
    import torch
    g = hub_graph(list(degrees), 900)
    net = nd.Network(g, [nd.pqnode()] * g.nv, nd.piline())
    on = O.OracleNetwork.from_batches(g.nv, g.src, g.dst, [m.kind for m in net.vertex_batches], net.vertex_batch,
                                      [(O.E_PILINE, O.C_FIDUCIAL)], net.edge_batch)
    rng = np.random.default_rng(len(degrees))
    u, p = rng.normal(size=net.dim).astype(dtype), rng.uniform(0.5, 1.5, size=net.pdim).astype(dtype)
    got = gpu_rhs(nd.adapt(net, torch.float64 if dtype == np.float64 else torch.float32), u, p, cuda, dtype)
    ref = on.rhs(u.astype(np.float64), p.astype(np.float64))
    rows = np.flatnonzero(g.degree())
    at = np.stack([2 * rows, 2 * rows + 1])
    if dtype == np.float64:
        np.testing.assert_array_equal(got[at], ref[at])
        return
    # du = S / conj(i): the relative error of |i|, whose n currents (|V| <= 5, 1 / |Z| <= 1.5) sum to
    # |i| with an error of n (n + 8) 2^-24 * 10, and 16 roundings of the division
    n, s = g.degree()[rows], np.hypot(*p[:2 * g.nv].astype(np.float64).reshape(-1, 2)[rows].T)
    size = np.hypot(*ref[at])
    current = s / size
    assert np.all(np.hypot(*(got[at].astype(np.float64) - ref[at])) <= size * (n * (n + 8.0) * 10 / current + 16) * 2.0 ** -24)
