"""Per-cluster evaluation (csrc/ck_direct.cu) of many clusters in one call
against the same clusters one at a time by the oracle: block remainders, mixed
and excluded types, distances at and beyond the outer cutoffs and below the
inner ones, every power count of the fixed-point form, and a set without its streams.
Tolerance: the FP64 form's gates, relative to the largest value where the
extrapolation below the inner cutoff makes it large."""

import numpy as np
import pytest

from conftest import E_REL_TOL

pytestmark = pytest.mark.gpu


def clusters(rng, n, body, ntypes, lo, hi):
    x = np.zeros((n, body, 3))
    i, j = np.triu_indices(body, 1)
    for c in range(n):
        while True:
            x[c] = rng.uniform(0.0, hi / 1.5, (body, 3))
            r = np.linalg.norm(x[c][j] - x[c][i], axis=1)
            if r.min() > lo:
                break
    dr = x[:, j] - x[:, i]
    return np.linalg.norm(dr, axis=2), dr, rng.integers(0, ntypes, (n, body))


@pytest.mark.parametrize("body,orders", [(3, (6, 2, 0)), (3, (6, 5, 0)), (3, (12, 11, 0)), (4, (6, 3, 2)), (4, (6, 3, 3)),
                                         (4, (8, 4, 4)), (4, (6, 3, 5)), (3, (6, 12, 0))], ids=str)
@pytest.mark.parametrize("n", [1, 7, 333])
def test_batch_matches_oracle(tmp_path, native_lib, body, orders, n):
    from chimes_calculator_gb300 import Calculator, synth
    from oracle.oracle import Oracle
    spec = synth.ParamSpec(elements=["C", "N"], orders=orders, rin=1.2, rout=5.0, lam=(1.3, 1.6),
                           fcut=("CUBIC",) if orders[1] == 5 else ("TERSOFF", 0.5), s3max=4.0, s4max=3.6,
                           excluded3=(1,), excluded4=(1,),
                           seed=90 + sum(orders))
    path = synth.write_param_file(str(tmp_path / "p.txt"), spec)
    rng = np.random.default_rng(3 * n + body)
    dx, dr, typ = clusters(rng, n, body, 2, 1.0, 4.4 if body == 3 else 3.8)
    if n > 1:
        dx[0, 0] = 4.0 if body == 3 else 3.6   # the outer cutoff itself: dropped
    c = Calculator()
    c.load_params(path)
    got = c.clusters(body, dx, dr, typ)
    o = Oracle(path)
    want = {k: np.zeros_like(got[k]) for k in ("energy", "force", "stress")}
    fn = o.compute_3b if body == 3 else o.compute_4b
    for q in range(n):
        want["energy"][q] = fn(dx[q], dr[q], typ[q], want["force"][q], want["stress"][q], 0.0)
    assert n == 1 or np.count_nonzero(want["energy"]) >= n // 2
    for k, v in want.items():
        assert np.abs(got[k] - v).max() <= 10 * E_REL_TOL * max(1.0, np.abs(v).max()), k
