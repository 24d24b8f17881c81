"""The RHS at the sizes where its kernels change: the fused launch of small networks and the
two-phase layout above it, rows on both sides of the degree limits (a thread in a window, the
heavy kernel or a block of the fused launch)."""
import numpy as np
import pytest

import nd_gb300 as nd
from oracle import oracle as O

from ndtest import gpu_rhs, random_inputs

pytestmark = pytest.mark.gpu

VM = {O.V_DIFFUSION: nd.diffusion_vertex, O.V_SWING: nd.kuramoto_second}
EM = {O.E_DIFFUSION: nd.diffusion_edge, O.E_KURAMOTO: nd.static_line}


def hubs(degrees, nv):
    """Vertices 0, 1, ... with the given degrees into the rest, and a path through the rest."""
    k = len(degrees)
    e = [(h, k + i) for h, d in enumerate(degrees) for i in range(d)] + [(i, i + 1) for i in range(k, nv - 1)]
    arr = np.array(sorted(e), dtype=np.int64)
    return nd.Graph(nv, np.ascontiguousarray(arr[:, 0]), np.ascontiguousarray(arr[:, 1]))


@pytest.mark.parametrize("graph", [
    lambda: nd.cycle_graph(3),                                  # one window
    lambda: hubs([32, 33, 128, 129, 255, 256, 257], 700),       # fused: window / heavy rows
    lambda: hubs([511, 512, 513, 1024, 1025, 2047, 2048, 2049, 2500], 6000),  # tiles of the block scan
    lambda: nd.barabasi_albert(262_000, 4, seed=3),             # just below the FP64 fused limit
    lambda: nd.barabasi_albert(263_000, 4, seed=3),             # just above it
], ids=["cycle3", "hubs257", "hubs2500", "below", "above"])
@pytest.mark.parametrize("vk,ek", [(O.V_DIFFUSION, O.E_DIFFUSION), (O.V_SWING, O.E_KURAMOTO)])
def test_rhs_at_layout_limits(cuda, graph, vk, ek):
    """Diffusion has the oracle's bits (no sine); with sines 1e-13 of the term scale, as the
    other parity tests; FP32 within 4e-6 of it (24 eps of a compensated sum)."""
    g = graph()
    on = O.OracleNetwork.from_graph(g, vk, ek)
    u, p = random_inputs(on, vk, np.random.default_rng(g.nv))
    net = nd.Network(g, VM[vk](), EM[ek]())
    import torch
    got, ref = gpu_rhs(nd.adapt(net, torch.float64), u, p, cuda, np.float64), on.rhs(u, p)
    scale = on.abs_terms(u, p) + np.abs(ref)
    if ek == O.E_DIFFUSION:
        np.testing.assert_array_equal(got, ref)
    else:
        assert np.all(np.abs(got - ref) <= 1e-13 * scale)
    u32, p32 = u.astype(np.float32), p.astype(np.float32)
    ref = on.rhs(u32.astype(np.float64), p32.astype(np.float64))
    got = gpu_rhs(nd.adapt(net, torch.float32), u32, p32, cuda, np.float32)
    scale = on.abs_terms(u32.astype(np.float64), p32.astype(np.float64)) + np.abs(ref)
    assert np.all(np.abs(got - ref) <= 4e-6 * scale)


@pytest.mark.parametrize("ne,dtype", [
    (2_100_001, np.float64), (2_100_002, np.float64), (2_100_003, np.float64), (2_100_000, np.float32),
    (2_100_003, np.float32), (2_100_004, np.float32),            # every remainder of four edges per thread
    (96 * 2**17 - 1, np.float64), (96 * 2**17, np.float64), (96 * 2**17 + 1, np.float64),  # 96 MiB of edge values
])
@pytest.mark.parametrize("nv", [300_000, 300_001])  # edge parameters on and off a 16-byte boundary
def test_two_phase_edge_values(cuda, ne, dtype, nv):
    """Rows that gather from the edge values or from their grouped copy against the fused layout:
    the same bits in FP64; FP32 within 4e-6 of the term scale of either (24 eps of a compensated
    sum), so within twice that of each other."""
    import torch
    rng = np.random.default_rng(ne + nv)
    a, b = rng.integers(0, nv, size=(2, ne + ne // 8))
    key = np.unique(np.minimum(a, b)[a != b] * np.int64(nv) + np.maximum(a, b)[a != b])
    assert key.size >= ne
    key = np.sort(rng.permutation(key)[:ne])
    src, dst = np.ascontiguousarray(key // nv), np.ascontiguousarray(key % nv)
    net = nd.adapt(nd.Network(nd.Graph(nv, src, dst), nd.diffusion_vertex(), nd.diffusion_edge()),
                   torch.float64 if dtype == np.float64 else torch.float32)
    u, p = rng.normal(size=nv).astype(dtype), rng.uniform(0.5, 1.5, size=ne).astype(dtype)
    net.set_layout("auto")
    auto = gpu_rhs(net, u, p, cuda, dtype)
    # 2.1e6 edges are the last that FP32 takes in one launch
    assert net.kernel_times()["edge_phase"][0] == (0 if dtype == np.float32 and ne == 2_100_000 else 1)
    net.set_layout("fused")
    fused = gpu_rhs(net, u, p, cuda, dtype)
    if dtype == np.float64:
        np.testing.assert_array_equal(auto, fused)
    else:
        term = np.abs(p.astype(np.float64) * (u[src].astype(np.float64) - u[dst]))
        scale = np.bincount(src, term, nv) + np.bincount(dst, term, nv)
        assert np.all(np.abs(auto.astype(np.float64) - fused) <= 8e-6 * scale)


@pytest.mark.parametrize("degrees", [(8192,), (8193,), (20_000, 8193, 8192, 129, 128), (9000, 8500, 8193)])
@pytest.mark.parametrize("vk,ek", [(O.V_DIFFUSION, O.E_DIFFUSION), (O.V_SWING, O.E_KURAMOTO)])
def test_f32_hubs_of_small_networks(cuda, degrees, vk, ek):
    """Rows above 8192 terms in the heavy kernel, shorter ones in the fused launch: every row within
    4e-6 of the FP64 oracle's term scale (24 eps of a compensated sum), and the heavy kernel
    runs where such a row is there."""
    g = hubs(list(degrees), 21_000)
    on = O.OracleNetwork.from_graph(g, vk, ek)
    u, p = random_inputs(on, vk, np.random.default_rng(len(degrees)), np.float32)
    import torch
    nw = nd.adapt(nd.Network(g, VM[vk](), EM[ek]()), torch.float32)
    got, ref = gpu_rhs(nw, u, p, cuda, np.float32), on.rhs(u.astype(np.float64), p.astype(np.float64))
    assert np.all(np.abs(got - ref) <= 4e-6 * (on.abs_terms(u.astype(np.float64), p.astype(np.float64)) + np.abs(ref)))
    assert nw.kernel_times()["heavy_rows"][0] == int(max(degrees) > 8192)


@pytest.mark.parametrize("long_rows", [1, 3, 4, 5, 6, 31, 40])  # marked by their warp up to four, by a thread above
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_windows_of_long_rows(cuda, long_rows, dtype):
    """Windows with few and with many rows above 32 terms: the oracle's bits in FP64, FP32 within 4e-6
    of the term scale."""
    import torch
    g = hubs([33 + 7 * i % 60 for i in range(long_rows)], 1500)
    on = O.OracleNetwork.from_graph(g, O.V_DIFFUSION, O.E_DIFFUSION)
    u, p = random_inputs(on, O.V_DIFFUSION, np.random.default_rng(long_rows), dtype)
    nw = nd.adapt(nd.Network(g, nd.diffusion_vertex(), nd.diffusion_edge()),
                  torch.float64 if dtype == np.float64 else torch.float32)
    got, ref = gpu_rhs(nw, u, p, cuda, dtype), on.rhs(u.astype(np.float64), p.astype(np.float64))
    if dtype == np.float64:
        np.testing.assert_array_equal(got, ref)
    else:
        assert np.all(np.abs(got - ref) <= 4e-6 * on.abs_terms(u.astype(np.float64), p.astype(np.float64)))


@pytest.mark.parametrize("order", ["sequential", "sequential_hw"])
@pytest.mark.parametrize("first", [257, 509, 1023])  # remainders of 16 terms; the ends of a tile
def test_heavy_row_remainders(cuda, first, order):
    """Heavy rows of every remainder, by the scan and by hardware adds: the oracle's bits."""
    import torch
    g = hubs([first + i for i in range(18)], 1500)
    on = O.OracleNetwork.from_graph(g, O.V_DIFFUSION, O.E_DIFFUSION)
    u, p = random_inputs(on, O.V_DIFFUSION, np.random.default_rng(first))
    nw = nd.adapt(nd.Network(g, nd.diffusion_vertex(), nd.diffusion_edge()), torch.float64)
    nw.set_sum_order(order)
    np.testing.assert_array_equal(gpu_rhs(nw, u, p, cuda, np.float64), on.rhs(u, p))
