"""The mixed form's tensor-core contractions (csrc/ck_tensor.cu) against the
oracle: every width of both body orders, buckets from one cluster to more tiles
than one CTA's groups take at a time, with the pair-table cache (s4max below s3max)
and without it (4-body cutoff above the 3-body one), and pairs below the inner
cutoff.  Tolerance: the mixed form's own gates."""

import numpy as np
import pytest

from conftest import MIXED_E_REL_TOL, MIXED_S_ABS_TOL, mixed_force_tol

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cuts", [(4.0, 3.4), (3.4, 3.8)], ids=["cache", "nocache"])
@pytest.mark.parametrize("o3,o4", [(2, 2), (3, 3), (4, 4), (5, 2), (6, 3), (7, 4), (8, 2), (9, 3), (10, 4), (11, 4)])
@pytest.mark.parametrize("n,rin", [(5, 0.9), (48, 1.5), (300, 0.9)])
def test_widths_and_remainders(tmp_path, native_lib, cuts, o3, o4, n, rin):
    from chimes_calculator_gb300 import MIXED, Calculator, synth
    from oracle.oracle import Oracle
    if rin > 1.0 and o3 > 8:
        pytest.skip("sums of high orders extrapolated below the inner cutoff exceed the gates in FP32")
    spec = synth.ParamSpec(elements=["C", "N"], orders=(12, o3, o4), rin=rin, rout=5.0, lam=(1.3, 1.6),
                           fcut=("CUBIC",) if o3 == 5 else ("TERSOFF", 0.5), s3max=cuts[0], s4max=cuts[1],
                           seed=61 + o3)
    path = synth.write_param_file(str(tmp_path / "p.txt"), spec)
    side = (n / 0.09) ** (1.0 / 3.0)
    cfg = synth.random_config(n, np.diag([side] * 3), ["C", "N"], 1.0, seed=17 + n)
    ref = Oracle(path).calculate(cfg.pos, cfg.types, cfg.cell)
    c = Calculator(precision=MIXED)
    c.set_contraction(4)
    c.load_params(path)
    got = c.evaluate(cfg.pos, cfg.types, cfg.cell)
    assert c.tuning()["tc3"] == 1 and c.tuning()["tc4"] == 1
    big = max(1.0, np.abs(ref["stress"]).max())
    assert abs(got["energy"] - ref["energy"]) <= MIXED_E_REL_TOL * max(1.0, abs(ref["energy"]))
    assert np.abs(got["force"] - ref["force"]).max() <= mixed_force_tol(np.abs(ref["force"]).max())
    assert np.abs(got["stress"] - ref["stress"]).max() <= MIXED_S_ABS_TOL * big


def test_small_batch_takes_the_faster_form(tmp_path, native_lib):
    """Autotuning with the tensor cores asked for takes the fastest 3-body form it timed,
    in a batch of a few tiles too: the tensor-core kernel needs less than half of the
    per-coefficient kernels' time for these 60 thousand triplets, 1.5 is allowed."""
    import ctypes

    from chimes_calculator_gb300 import MIXED, Calculator, synth
    spec = synth.ParamSpec(elements=["C", "N"], orders=(12, 10, 4), rin=0.9, rout=5.0, lam=1.4, s3max=4.0, s4max=3.4,
                           seed=61)
    path = synth.write_param_file(str(tmp_path / "p.txt"), spec)
    side = (110 / 0.09) ** (1.0 / 3.0)
    cfgs = [synth.random_config(110, np.diag([side] * 3), ["C", "N"], 1.0, seed=17 + k) for k in range(11)]
    ms = {}
    for tuned in (True, False):
        c = Calculator(precision=MIXED)
        c.set_contraction(4)
        c.load_params(path)
        packed = c.pack([(q.pos, q.types, q.cell) for q in cfgs])
        if tuned:
            c.autotune(packed)
        c.stage(packed)
        t, n, k = (ctypes.c_double * 4)(), ctypes.c_longlong(), ctypes.c_int()
        for _ in range(2):   # (the first launches size the lists)
            c.lib.ck_set_profiling(c.h, 1)
            for _ in range(10):
                c.launch()
                c.lib.ck_read_stage_times(c.h, t, ctypes.byref(n), ctypes.byref(k))
                c.collect()
        ms[tuned] = t[2] / n.value
    assert ms[True] <= 1.5 * ms[False], ms
