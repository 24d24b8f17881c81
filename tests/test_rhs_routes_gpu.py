"""The right-hand side on the routes that only large networks take, each named by the kernels that
ran: rows beside or after the edge phase, gathering from the edge values or their grouped copy."""
import numpy as np
import pytest

import nd_gb300 as nd
from oracle import oracle as O

from ndtest import gpu_rhs, random_inputs

pytestmark = pytest.mark.gpu

VM = {O.V_DIFFUSION: nd.diffusion_vertex, O.V_SWING: nd.kuramoto_second, O.V_KURAMOTO: nd.kuramoto_first}
EM = {O.E_DIFFUSION: nd.diffusion_edge, O.E_KURAMOTO: nd.static_line}
MODELS = [(O.V_DIFFUSION, O.E_DIFFUSION), (O.V_SWING, O.E_KURAMOTO)]


def canonical(nv, src, dst):
    order = np.lexsort((dst, src))
    return nd.Graph(nv, np.ascontiguousarray(src[order]), np.ascontiguousarray(dst[order]))


def check(cuda, g, vk, ek, dtype, route):
    """FP64: the oracle's bits without a sine, else 1e-13 of the rows' terms; FP32: 4e-6 of them (24
    eps of a compensated sum), with the inputs as rounded.  Then twelve calls in a row, each on
    states of its own, have the bits of calls made one at a time.  `route`: launches by kernel."""
    import torch
    on = O.OracleNetwork.from_graph(g, vk, ek)
    u, p = random_inputs(on, vk, np.random.default_rng(g.ne % 1000))
    u, p = u.astype(dtype), p.astype(dtype)
    nw = nd.adapt(nd.Network(g, VM[vk](), EM[ek]()), torch.float64 if dtype == np.float64 else torch.float32)
    got = gpu_rhs(nw, u, p, cuda, dtype)
    assert {k: n for k, (n, _) in nw.kernel_times().items() if n} == route
    u64, p64 = u.astype(np.float64), p.astype(np.float64)
    ref = on.rhs(u64, p64)
    if dtype == np.float64 and ek == O.E_DIFFUSION:
        np.testing.assert_array_equal(got, ref)
    else:
        bound = (1e-13 if dtype == np.float64 else 4e-6) * (on.abs_terms(u64, p64) + np.abs(ref))
        assert np.all(np.abs(got.astype(np.float64) - ref) <= bound)
    x = torch.from_numpy(u).to(cuda)
    us = torch.stack([torch.roll(x, 2 * i) for i in range(12)])
    pt = torch.from_numpy(p).to(cuda)
    alone, row = torch.empty_like(us), torch.empty_like(us)
    for i in range(12):
        nw(alone[i], us[i], pt, 0.0)
        torch.cuda.synchronize()
    for i in range(12):
        nw(row[i], us[i], pt, 0.0)
    assert torch.equal(row, alone)


@pytest.mark.parametrize("vk,ek", MODELS)
@pytest.mark.parametrize("n,k", [(2100, 2002), (3000, 1500)])  # 2,102,100 and 2,250,000 edges
def test_f32_dense_rows(cuda, n, k, vk, ek):
    """FP32 rows of a dense network, a warp each, beside the edge phase's last blocks."""
    check(cuda, nd.watts_strogatz(n, k, 0.2, seed=5), vk, ek, np.float32, {"edge_phase": 1, "row_phase": 1})


def hubs_and_path(degrees, nv):
    k = len(degrees)
    src = np.concatenate([np.full(d, h) for h, d in enumerate(degrees)] + [np.arange(k, nv - 1)]).astype(np.int64)
    dst = np.concatenate([k + np.arange(d) for d in degrees] + [np.arange(k + 1, nv)]).astype(np.int64)
    return canonical(nv, src, dst)


@pytest.mark.parametrize("vk,ek", MODELS)
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_hubs_of_networks_in_two_launches(cuda, dtype, vk, ek):
    """Rows on both sides of every limit: 32 terms (a thread), 128 (FP32: a warp), 2048 (the heavy
    kernel; FP64 from 129 on at this size)."""
    degrees = [31, 32, 33, 127, 128, 129, 130, 512, 1000, 2047, 2048, 2049, 2050, 3000, 20_000]
    check(cuda, hubs_and_path(degrees, 2_150_000), vk, ek, dtype, {"edge_phase": 1, "row_phase": 1, "heavy_rows": 1})


def banded(nv, k, sparse, spread):
    """`sparse` sources 12 vertices apart with one edge each to the far end (a chunk of edges spans
    thousands of vertices, and every bucket of destinations but the last is empty); `spread` sources of
    0 to 4 edges to anywhere behind them (chunks that fill every bucket); then vertices with
    edges to the k behind them (chunks of one bucket)."""
    rng = np.random.default_rng(nv + k)
    s = [12 * np.arange(sparse)]
    d = [nv - 1 - np.arange(sparse) % 1000]
    lo = 12 * sparse
    deg = rng.integers(0, 5, spread)
    deg[::7] = 0
    ss = np.repeat(lo + np.arange(spread), deg)
    key = np.unique(ss * np.int64(nv) + rng.integers(lo + spread, nv, ss.size))
    s.append(key // nv)
    d.append(key % nv)
    first = lo + spread
    b = np.repeat(np.arange(first, nv - k), k)
    s.append(b)
    d.append(b + 1 + np.tile(np.arange(k), nv - k - first))
    return canonical(nv, np.concatenate(s).astype(np.int64), np.concatenate(d).astype(np.int64))


@pytest.mark.parametrize("vk,ek", MODELS[:1])
@pytest.mark.parametrize("nv,k,grouped", [(160_000, 24, False), (300_001, 72, True)])
def test_edge_chunks_of_every_shape(cuda, nv, k, grouped, vk, ek):
    """The edge kernels on chunks whose sources lie far apart, whose destinations fill every bucket, and
    that lie in one bucket: with the rows gathering from the edge values, and from their grouped copy
    (above 96 MiB of them)."""
    g = banded(nv, k, 5000, 30_000)
    assert (8 * g.ne > 96 * 2**20) == grouped and g.ne > 1_050_000
    check(cuda, g, vk, ek, np.float64, {"edge_phase": 1, "row_phase": 1})
