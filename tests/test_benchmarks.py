"""The benchmarks report no figure over states that are not solutions, and a leg that fails costs
only itself."""
import importlib.util
from pathlib import Path

import numpy as np
import pytest

import nd_gb300.benchmarks as NB

ROOT = Path(__file__).resolve().parent.parent


def bench():
    spec = importlib.util.spec_from_file_location("bench", ROOT / "bench.py")
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


def test_states_that_are_not_solutions():
    u, offset = np.arange(9.0), np.array([0, 2, 3, 9])
    NB.require_solved("solve", u, offset, np.zeros(3, np.int32))
    with pytest.raises(RuntimeError, match="1 instances not solved, first 2"):
        NB.require_solved("solve", u, offset, np.array([0, 0, -5]))
    for bad, first in ((0, 0), (2, 1), (8, 2)):
        v = u.copy()
        v[bad] = np.nan if bad else np.inf
        with pytest.raises(RuntimeError, match=f"not finite, first {first}"):
            NB.require_solved("solve", v, offset, np.zeros(3, np.int32))


def test_a_failing_leg_leaves_the_line(monkeypatch):
    b, line = bench(), {"value": 1.0}

    def fails(n):
        raise RuntimeError("steady states: 1 instances with a state that is not finite, first 542")

    monkeypatch.setattr(NB, "ensemble", fails)
    b.secondary_leg(line, "ensemble", b.ensemble_leg)
    b.secondary_leg(line, "other", lambda: {"x": 2})
    assert line == {"value": 1.0, "ensemble": {"error": "RuntimeError: steady states: 1 instances with a state that "
                                                        "is not finite, first 542"}, "other": {"x": 2}}
