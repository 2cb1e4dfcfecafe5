"""The FP64 form's fixed-point contraction (csrc/ck_fixed.cu) against the
oracle: every power count its kernels are instantiated for and those between,
every warps-per-tile setting, bucket remainders from one cluster to a few
tiles, pairs below the inner cutoff (tables scaled down by a power of two), and
coefficients of very uneven size.

Tolerance: the FP64 form's own gates (1e-10 of the energy, 1e-9 absolute force
and stress), relative to the largest force where the penalty region makes
forces large; the format's roundings are 2^-57 of full scale, below FP64's."""

import numpy as np
import pytest

from conftest import E_REL_TOL, F_ABS_TOL, S_ABS_TOL

pytestmark = pytest.mark.gpu


def check(path, cfg, tuning=None, contraction=1):
    from chimes_calculator_gb300 import Calculator
    from oracle.oracle import Oracle
    ref = Oracle(path).calculate(cfg.pos, cfg.types, cfg.cell)
    c = Calculator()
    c.set_contraction(contraction)
    if tuning:
        c.set_tuning(*tuning)
    c.load_params(path)
    got = c.evaluate(cfg.pos, cfg.types, cfg.cell)
    assert c.tuning()["fact3"] == 1
    big = max(1.0, np.abs(ref["force"]).max())
    assert abs(got["energy"] - ref["energy"]) <= E_REL_TOL * max(1.0, abs(ref["energy"]))
    assert np.abs(got["force"] - ref["force"]).max() <= F_ABS_TOL * big
    assert np.abs(got["stress"] - ref["stress"]).max() <= S_ABS_TOL * big


@pytest.mark.parametrize("orders", [(4, 2, 2), (6, 4, 3), (6, 5, 4), (8, 8, 5), (8, 9, 2), (12, 10, 4), (12, 11, 3)],
                         ids=lambda o: "%d-%d" % o[1:])
@pytest.mark.parametrize("n", [5, 48])
def test_orders_and_remainders(tmp_path, native_lib, orders, n):
    from chimes_calculator_gb300 import synth
    spec = synth.ParamSpec(elements=["C", "N"], orders=orders, rin=0.9, rout=4.4, lam=(1.2, 1.6),
                           fcut=("CUBIC",) if orders[1] == 5 else ("TERSOFF", 0.5), s3max=4.0, s4max=3.4,
                           expand=orders[1] == 4, seed=31 + orders[1])
    path = synth.write_param_file(str(tmp_path / "p.txt"), spec)
    side = (n / 0.09) ** (1.0 / 3.0)
    check(path, synth.random_config(n, np.diag([side] * 3), ["C", "N"], 1.0, seed=7 + n))


@pytest.mark.parametrize("warps", [1, 2, 4])
@pytest.mark.parametrize("contraction", [1, 2], ids=["cache", "nocache"])
def test_below_inner_cutoff(tmp_path, native_lib, warps, contraction):
    """A fifth of the pairs lie below the inner cutoff, one as close as 0.5 of it."""
    from chimes_calculator_gb300 import synth
    spec = synth.ParamSpec(elements=["C", "N"], orders=(8, 6, 4), rin=1.5, rout=4.4, lam=1.4, s3max=4.0, s4max=3.4,
                           penalty=(0.02, 100.0), seed=77)
    path = synth.write_param_file(str(tmp_path / "p.txt"), spec)
    cfg = synth.random_config(40, np.diag([7.6, 7.6, 7.6]), ["C", "N"], 0.8, seed=3)
    check(path, cfg, (warps, warps, 4), contraction)


def test_uneven_coefficients(tmp_path, native_lib):
    """One coefficient of a tuple 10^6 times the others (amplitude by the largest,
    not by the sum)."""
    from chimes_calculator_gb300 import synth
    spec = synth.ParamSpec(elements=["C", "N"], orders=(6, 4, 3), rin=0.9, rout=4.4, lam=1.4, s3max=4.0, s4max=3.4,
                           seed=5)
    out, block, row = [], None, 0
    for ln in synth.build_param_text(spec).split("\n"):
        t = ln.split()
        if ln.startswith(("TRIPLETTYPE", "QUADRUPLETYPE")):
            block, row = ln.split()[0], 0
        elif block and len(t) in (7, 10) and t[0].isdigit():
            if row == 2:
                t[-1] = repr(1e6 * float(t[-1]))
            row += 1
            ln = " ".join(t)
        out.append(ln)
    path = str(tmp_path / "p.txt")
    with open(path, "w") as f:
        f.write("\n".join(out))
    check(path, synth.random_config(40, np.diag([7.6, 7.6, 7.6]), ["C", "N"], 1.0, seed=3))
