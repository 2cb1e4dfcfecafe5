"""A captured graph is replayed only while every buffer it works on stays where
it was: small batches between two evaluations of one large configuration grow
the per-configuration arrays (bounding boxes) and no other, so the large one's
graph is captured again and its results stay."""

import numpy as np
import pytest

from conftest import E_REL_TOL, F_ABS_TOL

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count,n", [(12, 8), (16, 16), (200, 8)])
def test_small_batch_between_replays(golden, native_lib, count, n):
    from chimes_calculator_gb300 import Calculator, synth
    g = golden["c2"]
    c = Calculator(graph=True)
    c.load_params(g.params)
    el = sorted(set(g.cfg.types))
    side = (n / 0.05) ** (1.0 / 3.0)
    small = [synth.random_config(n, np.diag([side] * 3), el, 1.2, seed=k) for k in range(count)]
    small = [(s.pos, s.types, s.cell) for s in small]

    def large():
        r = c.evaluate(g.cfg.pos, g.cfg.types, g.cfg.cell)
        assert abs(r["energy"] - g.energy) <= E_REL_TOL * abs(g.energy)
        assert np.abs(r["force"] - g.force).max() <= F_ABS_TOL
    for _ in range(4):
        large()
    captured = c.graph_captures()
    assert captured >= 1
    large()
    assert c.graph_captures() == captured   # replayed
    first = c.evaluate_batch(small)
    for _ in range(3):
        large()
    assert c.graph_captures() > captured    # not the graph of the old buffers
    again = c.evaluate_batch(small)
    for a, b in zip(first, again):
        assert abs(a["energy"] - b["energy"]) <= E_REL_TOL * max(1.0, abs(a["energy"]))
        assert np.abs(a["force"] - b["force"]).max() <= F_ABS_TOL
