"""Batched steady states of swing networks whose solve must not be taken for a solution, and of
networks that are not connected."""
import numpy as np
import pytest

import nd_gb300 as nd
from nd_gb300 import _capi as capi
from nd_gb300.ensemble import Ensemble

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
