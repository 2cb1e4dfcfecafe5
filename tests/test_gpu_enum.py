"""The cluster enumeration (csrc/ck_lists.cu) at the bucket counts that its blocks
keep in shared memory, and past them."""

import numpy as np
import pytest

from conftest import E_REL_TOL, F_ABS_TOL, S_ABS_TOL

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_sets", [2, 3, 4], ids=["640", "960", "1280"])
def test_bucket_counts(tmp_path, native_lib, n_sets):
    """640, 960 and 1280 buckets (1024 fit a block's shared memory), with enough
    atoms that one warp works on an atom: the results of a handle with one set."""
    from chimes_calculator_gb300 import Calculator, synth
    el = ["C", "H", "N", "O"]
    spec = synth.ParamSpec(elements=el, orders=(4, 2, 2), rin=0.9, rout=4.4, lam=1.4, s3max=3.6, s4max=3.0, seed=21)
    path = synth.write_param_file(str(tmp_path / "p.txt"), spec)
    cfgs = [synth.random_config(100, np.diag([11.0, 11.0, 11.0]), el, 1.0, seed=k) for k in range(4)] * 26
    cfgs = [(c.pos, c.types, c.cell) for c in cfgs]
    one, many = Calculator(), Calculator()
    one.load_params(path)
    for _ in range(n_sets):
        many.load_params(path)
    ref = one.evaluate_batch(cfgs[:4])
    got = many.evaluate_batch(cfgs, slots=[k % n_sets for k in range(len(cfgs))])
    for k, r in enumerate(got):
        e = ref[k % 4]
        assert abs(r["energy"] - e["energy"]) <= E_REL_TOL * max(1.0, abs(e["energy"]))
        assert np.abs(r["force"] - e["force"]).max() <= F_ABS_TOL
        assert np.abs(r["stress"] - e["stress"]).max() <= S_ABS_TOL
