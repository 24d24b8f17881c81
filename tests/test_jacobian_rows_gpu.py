"""The Jacobian values and the JVP on rows at the lengths where their kernels change (a thread, a
warp or a block per row), with and without repeated edges (which keep the searching kernels)."""
import numpy as np
import pytest

import nd_gb300 as nd
from oracle import oracle as O

from test_batched_gpu import ALL_EDGES, VKINDS, build
from test_jacobian_gpu import check

pytestmark = pytest.mark.gpu


def wheel(leaves, repeated=False):
    """A hub with `leaves` neighbours, a ring through them, and an isolated last vertex; with
    `repeated`, the first edge of the hub twice."""
    e = [(0, i) for i in range(1, leaves + 1)] + [(i, i + 1) for i in range(1, leaves)] + [(1, leaves)]
    arr = np.array(sorted(e + e[:1] if repeated else e), dtype=np.int64)
    return nd.Graph(leaves + 2, np.ascontiguousarray(arr[:, 0]), np.ascontiguousarray(arr[:, 1]))


@pytest.mark.parametrize("leaves", [31, 32, 33, 70])
@pytest.mark.parametrize("repeated", [False, True])
def test_static_jacobian_rows(cuda, leaves, repeated):
    """Every static kind with every wrapper, all vertex kinds, against central differences."""
    g = wheel(leaves, repeated)
    rng = np.random.default_rng(leaves)
    edges = [b for b in ALL_EDGES if b[0] in (O.E_DIFFUSION, O.E_KURAMOTO)]
    net, on = build(g, VKINDS, edges, vassign=rng.integers(0, len(VKINDS), g.nv),
                    eassign=rng.integers(0, len(edges), g.ne))
    check(net, on, rng.normal(size=net.dim), rng.uniform(0.5, 1.5, size=net.pdim), cuda)


@pytest.mark.parametrize("leaves", [32, 33, 255, 256, 257, 1100])
@pytest.mark.parametrize("dtype,tol", [("float64", 1e-13), ("float32", 1e-5)])
def test_jvp_rows(cuda, leaves, dtype, tol):
    """nd_jvp against the assembled Jacobian: both sum at most 1100 terms of a row, in different
    orders, within tol of Σ |J| |v| (FP64: 1100 eps = 2.4e-13 at worst, a few eps in practice of
    the pairwise sums; FP32 likewise)."""
    import torch
    tdt = getattr(torch, dtype)
    g = wheel(leaves)
    net = nd.Network(g, nd.kuramoto_second(), nd.static_line())
    nw = nd.adapt(net, tdt)
    rng = np.random.default_rng(leaves)
    u, v = (torch.from_numpy(rng.normal(size=nw.dim)).to("cuda", tdt) for _ in range(2))
    p = torch.from_numpy(net.pflat(vertex={"Pm": rng.normal(size=g.nv)}, edge={"K": rng.uniform(5, 10, g.ne)}))
    p = p.to("cuda", tdt)
    jv = torch.empty_like(u)
    nd.jvp(nw, jv, u, p, v)
    J = nd.jacobian(nw, u, p).to_dense().double()
    scale = J.abs() @ v.double().abs()
    assert torch.all((J @ v.double() - jv.double()).abs() <= tol * (scale + 1e-300)).item()


def test_index_tensors_outlive_the_network(cuda):
    """A Jacobian asked for on a busy stream, whose network goes away before the stream gets to it: its
    index tensors are the pattern, although the memory of the network's own is free by then."""
    import torch
    g = nd.barabasi_albert(20_000, 2, seed=4)
    net = nd.Network(g, nd.kuramoto_second(), nd.static_line())
    u = torch.randn(net.dim, dtype=torch.float64, device=cuda)
    p = torch.rand(net.pdim, dtype=torch.float64, device=cuda) + 0.5
    nw = nd.adapt(net, torch.float64)
    ref = nd.jacobian(nw, u, p)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        torch.cuda._sleep(100_000_000)  # some 50 ms
    J = nd.jacobian(nw, u, p, stream=side)
    kept = [x.numel() for x in nw._jac_index[0]]
    nw._jac_index = None
    trash = [torch.full((n,), -1, dtype=torch.int64, device=cuda) for n in kept for _ in range(4)]
    torch.cuda.synchronize()
    assert trash[0][0].item() == -1
    assert torch.equal(J.crow_indices(), ref.crow_indices()) and torch.equal(J.col_indices(), ref.col_indices())
    assert torch.equal(J.values(), ref.values())


def test_stream_given_by_its_handle(cuda):
    """Any object with a cuda_stream attribute names the stream, as for the other calls."""
    import types

    import torch
    net = nd.Network(nd.watts_strogatz(50, 4, 0.2, seed=1), nd.kuramoto_first(), nd.kuramoto_edge())
    nw = nd.adapt(net, torch.float64)
    u = torch.randn(net.dim, dtype=torch.float64, device=cuda)
    p = torch.rand(net.pdim, dtype=torch.float64, device=cuda)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    J = nd.jacobian(nw, u, p, stream=types.SimpleNamespace(cuda_stream=side.cuda_stream))
    torch.cuda.synchronize()
    assert torch.equal(J.to_dense(), nd.jacobian(nw, u, p).to_dense())
