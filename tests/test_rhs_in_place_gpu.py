"""du over u: the RHS of the states that were there before the call."""
import numpy as np
import pytest

import nd_gb300 as nd

pytestmark = pytest.mark.gpu


def networks():
    ba, ws = nd.barabasi_albert(3000, 2, seed=1), nd.watts_strogatz(400, 6, 0.3, seed=2)
    return {
        "one launch": nd.Network(ws, nd.kuramoto_second(), nd.static_line()),
        "heavy rows": nd.Network(nd.barabasi_albert(60_000, 3, seed=3), nd.diffusion_vertex(), nd.diffusion_edge()),
        "two launches": nd.Network(nd.watts_strogatz(230_000, 20, 0.3, seed=4), nd.kuramoto_second(), nd.static_line()),
        "edge states": nd.Network(ba, nd.kuramoto_first(), nd.diffusion_odeedge()),
        "mixed": nd.Network(ws, [nd.kuramoto_first() if i % 2 else nd.kuramoto_second() for i in range(ws.nv)],
                            [nd.diffusion_odeedge() if i % 3 else nd.kuramoto_edge() for i in range(ws.ne)]),
        "power grid": nd.Network(ws, [nd.pqnode() if i % 3 else nd.generator() for i in range(ws.nv)], nd.piline()),
    }


@pytest.mark.parametrize("dtype", ["float64", "float32"])
@pytest.mark.parametrize("kind", ["one launch", "heavy rows", "two launches", "edge states", "mixed", "power grid"])
def test_du_is_u(cuda, kind, dtype):
    """The bits of a call with buffers of its own: in place, shifted by one entry, and captured."""
    import torch
    dt = getattr(torch, dtype)
    net = networks()[kind]
    nw = nd.adapt(net, dt)
    gen = torch.Generator(device=cuda).manual_seed(6)
    u = torch.randn(net.dim, dtype=dt, device=cuda, generator=gen)
    p = torch.rand(net.pdim, dtype=dt, device=cuda, generator=gen) + 0.5
    ref = torch.empty_like(u)
    nw(ref, u, p, 0.0)
    x = u.clone()
    nw(x, x, p, 0.0)
    assert torch.equal(x, ref)
    buf = torch.zeros(net.dim + 1, dtype=dt, device=cuda)
    for du, src in ((buf[:-1], buf[1:]), (buf[1:], buf[:-1])):
        src.copy_(u)
        nw(du, src, p, 0.0)
        assert torch.equal(du, ref)
    x.copy_(u)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        nw(x, x, p, 0.0)
    for _ in range(3):
        x.copy_(u)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(x, ref)
