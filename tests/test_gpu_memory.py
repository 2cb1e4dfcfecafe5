"""A configuration whose list fits the device but whose per-entry arrays (pair
tables, force scalars) do not is evaluated without them, with the same
results, on first use and when the lists outgrow their first estimate."""

import numpy as np
import pytest

from conftest import E_REL_TOL, F_ABS_TOL, MIXED_E_REL_TOL, mixed_force_tol

pytestmark = pytest.mark.gpu


def fill(leave):
    """Device memory taken except `leave` bytes."""
    import torch
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    return torch.empty(max(0, free - int(leave)), dtype=torch.uint8, device="cuda")


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("clumped", [False, True], ids=["uniform", "clumped"])
def test_without_entry_arrays(tmp_path, native_lib, precision, clumped):
    import torch
    from chimes_calculator_gb300 import FP64, MIXED, Calculator, synth
    spec = synth.ParamSpec(elements=["C", "N"], orders=(8, 8, 4), rin=0.9, rout=5.0, lam=1.4, s3max=4.0, s4max=3.2,
                           seed=31)
    path = synth.write_param_file(str(tmp_path / "p.txt"), spec)
    n = 24000
    side = (n / 0.09) ** (1.0 / 3.0)
    cfg = synth.random_config_batched(n, np.diag([side] * 3), ["C", "N"], 1.0, seed=4)
    cell = np.diag([side, side, side * (4.0 if clumped else 1.0)])   # clumped: three quarters of the cell empty
    args = (cfg.pos, cfg.types, cell)

    def calculator():
        c = Calculator(precision=FP64 if precision == "fp64" else MIXED)
        c.load_params(path)
        if precision == "mixed":
            c.set_contraction(4)
        return c
    c = calculator()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    want = c.evaluate(*args)
    used = free - torch.cuda.mem_get_info()[0]
    c.close()
    assert used > 300e6
    hog = fill(0.6 * used)
    try:
        c = calculator()
        for _ in range(2):
            got = c.evaluate(*args)
            e, f = (E_REL_TOL, F_ABS_TOL) if precision == "fp64" else (
                MIXED_E_REL_TOL, mixed_force_tol(np.abs(want["force"]).max()))
            assert abs(got["energy"] - want["energy"]) <= e * abs(want["energy"])
            assert np.abs(got["force"] - want["force"]).max() <= f
        small = synth.random_config(20, np.diag([7.0] * 3), ["C", "N"], 1.0, seed=5)
        alone = c.evaluate(small.pos, small.types, small.cell)
    finally:
        del hog
        torch.cuda.empty_cache()
    other = calculator().evaluate(small.pos, small.types, small.cell)
    assert abs(alone["energy"] - other["energy"]) <= MIXED_E_REL_TOL * max(1.0, abs(other["energy"]))
    assert np.abs(alone["force"] - other["force"]).max() <= mixed_force_tol(np.abs(other["force"]).max())
