"""Single 3- and 4-atom molecules in FP64 against sums in long double: the
fixed-point contraction's own error, which the gates of whole configurations
(1e-9) do not see.

The positions are multiples of 2^-20 and the cell's side is a power of two, so
that distances carry no error of the wrapping; the 2-body coefficients are
zero.  What remains is the error of the Morse variable and the cutoffs, common
to all forms, and the contraction's.

Tolerance: the mean error over 400 molecules against that of the per-coefficient
FP64 kernel on the same ones.  FP64 row and column sums have 1.21-1.23 (3-body;
their set-up multiplies by reciprocals) and 0.92-0.99 of it (4-body); 0.07 and 0.09
above that are allowed.  A contraction with sums cut at 2^-59 of full scale has
1.47 and 1.15."""

import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

L = np.longdouble
RIN, ROUT, LAM = 1.0, 5.0, 1.4


def parameters(body, orders, uneven):
    """Text of a one-element set without 2-body terms (4-body: nor 3-body ones) and its
    (powers, coefficient) rows; uneven: one coefficient 10^6 times the others."""
    from chimes_calculator_gb300 import synth
    spec = synth.ParamSpec(elements=["C"], orders=orders, rin=RIN, rout=ROUT, lam=LAM, fcut=("CUBIC",), s3max=4.4,
                           s4max=4.0, seed=11)
    out, rows, block = [], [], 0
    for ln in synth.build_param_text(spec).split("\n"):
        t = ln.split()
        for nb, head in ((2, "PAIRTYPE PARAMS"), (3, "TRIPLETTYPE"), (4, "QUADRUPLETYPE"), (0, "PAIRMAPS")):
            if ln.startswith(head):
                block = nb
        if block and t and t[0].isdigit() and len(t) == {2: 2, 3: 7, 4: 10}[block]:
            if block < body:
                t[-1] = "0.0"
            else:
                if uneven and len(rows) == 2:
                    t[-1] = repr(1e6 * float(t[-1]))
                rows.append((tuple(int(v) for v in t[1:-3]), float(t[-1])))
            ln = " ".join(t)
        out.append(ln)
    return "\n".join(out), rows


def forces(x, rows, rc):
    x = x.astype(L)
    slots = list(itertools.combinations(range(x.shape[1]), 2))
    lo, hi = np.exp(-L(rc) / L(LAM)), np.exp(-L(RIN) / L(LAM))
    d = [x[:, b] - x[:, a] for a, b in slots]
    r = [np.sqrt((v * v).sum(1)) for v in d]
    T, D, fc, fd = [], [], [], []
    for q in r:
        s = np.exp(-q / L(LAM))
        y, g = (s - (hi + lo) / 2) / ((lo - hi) / -2), -s / L(LAM) / ((lo - hi) / -2)
        t, u = [np.ones_like(y), y], [np.ones_like(y), 2 * y]
        for _ in range(2, max(max(p) for p, _ in rows) + 1):
            t.append(2 * y * t[-1] - t[-2])
            u.append(2 * y * u[-1] - u[-2])
        T.append(t)
        D.append([np.zeros_like(y)] + [n * u[n - 1] * g for n in range(1, len(t))])
        f0 = 1 - q / L(rc)
        fc.append(f0 ** 3)
        fd.append(-3 * f0 * f0 / L(rc))
    S, G = np.zeros(len(x), L), np.zeros((len(slots), len(x)), L)
    for p, c in rows:
        t = [T[q][p[q]] for q in range(len(slots))]
        S += L(c) * np.prod(t, axis=0)
        for q in range(len(slots)):
            G[q] += L(c) * np.prod([D[m][p[m]] if m == q else t[m] for m in range(len(slots))], axis=0)
    F = np.zeros(x.shape, L)
    for q, (a, b) in enumerate(slots):
        rest = np.prod([fc[m] for m in range(len(slots)) if m != q], axis=0) / r[q]
        f = (rest * (fc[q] * G[q] + fd[q] * S))[:, None] * d[q]
        F[:, a] += f
        F[:, b] -= f
    return F


@pytest.mark.parametrize("body,orders,uneven", [(3, (8, 10, 0), False), (3, (8, 4, 0), False), (3, (8, 10, 0), True),
                                                (4, (8, 2, 4), False), (4, (8, 2, 5), False), (4, (8, 2, 4), True)],
                         ids=["3b-10", "3b-4", "3b-uneven", "4b-4", "4b-5", "4b-uneven"])
def test_single_clusters(tmp_path, native_lib, body, orders, uneven):
    from chimes_calculator_gb300 import Calculator
    text, rows = parameters(body, orders, uneven)
    path = str(tmp_path / "p.txt")
    with open(path, "w") as f:
        f.write(text)
    rc = 4.4 if body == 3 else 4.0
    rng = np.random.default_rng(5)
    i, j = np.triu_indices(body, 1)
    x = np.zeros((400, body, 3))
    for m in range(len(x)):
        r = np.zeros(1)
        while r.min() <= RIN + 0.1 or r.max() >= rc - 0.1:
            x[m] = np.round(rng.uniform(5.0, 8.4, (body, 3)) * 2 ** 20) / 2 ** 20
            r = np.linalg.norm(x[m][j] - x[m][i], axis=1)
    want = forces(x, rows, rc)
    err = []
    for contraction in (1, 0):
        c = Calculator()
        c.set_contraction(contraction)
        c.load_params(path)
        got = np.array([g["force"] for g in c.evaluate_batch([(q, ["C"] * body, np.diag([16.0] * 3)) for q in x])])
        assert c.tuning()["fact%d" % body] == contraction
        err.append(float((np.abs(got - want).max((1, 2)) / np.abs(want).max((1, 2))).mean()))
    assert err[0] <= (1.3 if body == 3 else 1.08) * err[1], err
