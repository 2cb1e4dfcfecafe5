"""Cluster fingerprints on the GPU (the reference's FINGERPRINT build and its
histogram tool): the pair-style records (ck_nl_fingerprint) equal the
oracle's restatement of pair_chimes.cpp's, in order; the all-pairs
histogram (ck_fp_histogram) gives the oracle's counts; the frame workflow
(record -> combine -> histogram files) end to end; a large histogram keeps
its pair count."""

import os

import numpy as np
import pytest

from chimes_calculator_gb300 import fingerprint as fp
from chimes_calculator_gb300 import synth

pytestmark = pytest.mark.gpu

SKIN = 1.0


@pytest.fixture(scope="module")
def system(tmp_path_factory):
    from oracle.oracle import Oracle
    d = tmp_path_factory.mktemp("fp")
    spec = synth.ParamSpec(elements=["C", "N"], orders=(10, 6, 4), rin=0.9, rout=4.6, lam=(1.3, 1.6),
                           fcut=("TERSOFF", 0.5), s3max=3.8, s4max=3.0, excluded3=(2,), seed=5001)
    p = synth.write_param_file(str(d / "p.txt"), spec)
    o = Oracle(p)
    cfg = synth.random_config(160, np.diag([11.5, 11.5, 11.5]), ["C", "N"], 1.0, seed=5002)
    ti = o.type_indices(cfg.types)
    nl = synth.lammps_neighbors(cfg, ti, max(o.max_cutoffs) + SKIN, seed=5003)
    o.lammps_fingerprint(True)
    o.lammps_compute(nl, SKIN, rebuild=True)
    return p, o, nl


def _calc(p, nl):
    from chimes_calculator_gb300 import Calculator
    c = Calculator()
    c.load_params(p)
    c.nl_compute(nl, SKIN, rebuild=True)
    return c


@pytest.mark.parametrize("nb", [2, 3, 4])
def test_records_match_oracle(native_lib, system, nb):
    p, o, nl = system
    c = _calc(p, nl)
    d, t = c.nl_fingerprint(nb)
    od, ot = o.lammps_fp_records(nb)
    assert len(t) == len(ot) > 50
    assert np.array_equal(t, ot)
    assert np.array_equal(d, od)   # same FP64 distances, same order


@pytest.mark.parametrize("nb", [2, 3, 4])
def test_histogram_matches_oracle(native_lib, system, nb):
    p, o, nl = system
    c = _calc(p, nl)
    d, t = c.nl_fingerprint(nb)
    counts, ns = c.fp_histogram(nb, d, t)
    oc, ons = o.fp_histogram(nb, d, t)
    assert ns == ons == len(t) * (len(t) - 1) // 2
    assert np.array_equal(counts, oc)
    # two sets, and a bin count other than the tool's 100
    h = len(t) // 3
    counts, ns = c.fp_histogram(nb, d[:h], t[:h], d[h:], t[h:], nbin=37)
    oc, ons = o.fp_histogram(nb, d[:h], t[:h], d[h:], t[h:], nbin=37)
    assert ns == ons == h * (len(t) - h) and np.array_equal(counts, oc)


def test_frame_workflow(native_lib, system, tmp_path):
    """record_step -> combine_frames -> histogram_frames writes the tool's
    files; the histograms equal the oracle's on the same (6-digit) files."""
    p, o, nl = system
    c = _calc(p, nl)
    fp.record_step(c, 0, rank=0, directory=str(tmp_path))
    moved = synth.NeighborData(**{**nl.__dict__, "x": nl.x + np.random.default_rng(1).uniform(-0.1, 0.1, nl.x.shape)})
    c.nl_compute(moved, SKIN, rebuild=False)
    fp.record_step(c, 2, rank=0, directory=str(tmp_path))
    fp.combine_frames(str(tmp_path))
    res = fp.histogram_frames(c, str(tmp_path))
    assert sorted(res) == ["0", "2"]
    for fr in ("0", "2"):
        for nb in (2, 3, 4):
            assert os.path.exists(tmp_path / ("%s-%s.%db_clu-s.hist" % (fr, fr, nb)))
            d, t = fp.read_clusters(str(tmp_path / ("%s.all-%db-clusters.txt" % (fr, nb))), nb)
            oc, ons = o.fp_histogram(nb, d, t)
            counts, ns = res[fr][nb]
            assert ns == ons and np.array_equal(counts, oc)


def test_large_histogram_pair_count(native_lib, tmp_path):
    """C2-size 3-body records (1024 atoms): every pair j > i is counted once."""
    from chimes_calculator_gb300 import Calculator
    p = synth.write_param_file(str(tmp_path / "c2.txt"), synth.spec_c2())
    cfg = synth.config_c2()
    c = Calculator()
    c.load_params(p)
    nl = synth.lammps_neighbors(cfg, c.type_indices(cfg.types), max(c.info(0)["max_cutoffs"]) + SKIN, seed=7)
    c.nl_compute(nl, SKIN, rebuild=True)
    d, t = c.nl_fingerprint(3)
    n = len(t)
    assert n > 20000
    counts, ns = c.fp_histogram(3, d, t)
    assert ns == n * (n - 1) // 2 == counts.sum()


def test_errors(native_lib, system):
    from chimes_calculator_gb300 import ChimesError
    p, o, nl = system
    c = _calc(p, nl)
    d, t = c.nl_fingerprint(3)
    bad = t.copy()
    bad[0] = [0, 1, 1]   # triplet type 2 (C N N) is excluded in this set
    with pytest.raises(ChimesError, match="excluded"):
        c.fp_histogram(3, d, bad)
    with pytest.raises(ChimesError, match="nbin"):
        c.fp_histogram(3, d, t, nbin=5000)
    counts, ns = c.fp_histogram(3, d[:1], t[:1], d, t)   # one record in the first set: nothing counted
    assert ns == 0 and not counts.any()


@pytest.mark.parametrize("nb", [2, 3, 4])
@pytest.mark.parametrize("n1,n2", [(2, 0), (255, 0), (256, 1), (257, 0), (513, 0), (300, 513)])
@pytest.mark.parametrize("nbin", [1, 100, 1280])
def test_histogram_tile_edges(native_lib, system, nb, n1, n2, nbin):
    """Remainders of the 256 x 256 tiles and of a thread's two records, repeated
    records (distance zero), distances beyond the cutoffs, the smallest and the
    largest bin count: the oracle's counts exactly."""
    p, o, nl = system
    from chimes_calculator_gb300 import Calculator
    c = Calculator()
    c.load_params(p)
    rng = np.random.default_rng(1000 * nb + n1 + n2)

    def records(n):
        d = rng.uniform(0.8, 4.8, (n, nb * (nb - 1) // 2))
        t = np.zeros((n, nb), dtype=np.int32)   # one element: no excluded cluster type
        if n > 4:
            d[n // 2] = d[n // 4]
        return d, t
    s1 = records(n1)
    s2 = records(n2) if n2 else (None, None)
    counts, ns = c.fp_histogram(nb, *s1, *s2, nbin=nbin)
    oc, ons = o.fp_histogram(nb, *s1, *s2, nbin=nbin)
    assert ns == ons == (n1 * n2 if n2 else n1 * (n1 - 1) // 2)
    assert np.array_equal(counts, oc)


@pytest.mark.parametrize("nb", [2, 3, 4])
@pytest.mark.parametrize("many", [False, True])
def test_histogram_at_bin_edges(native_lib, system, nb, many):
    """Records whose distance to the first one crosses a bin edge within a few units
    in the last place of one of their distances: the counts follow the tool's
    host arithmetic exactly.  many: more such pairs than the device lists."""
    import math
    from chimes_calculator_gb300 import Calculator
    p, o, nl = system
    c = Calculator()
    c.load_params(p)
    npair = nb * (nb - 1) // 2
    rng = np.random.default_rng(40 + nb)
    nbin = 250
    maxd = 3.0 if nb == 2 else math.sqrt(12.0 if nb == 3 else 24.0) + 1.0
    w = maxd / nbin
    rout = o.max_cutoffs[nb - 2]   # (one cutoff per body order beyond pairs; a pair type's own is below)
    first = np.linspace(1.4, 0.8 * rout, npair)
    records = [first, first + 0.1]
    # the oracle's own counts locate the crossings: bin of (first, first with its last distance r)

    def bin_of(r):
        d = np.array([first, np.append(first[:-1], r)])
        return int(np.flatnonzero(o.fp_histogram(nb, d, np.zeros((2, nb), np.int32), nbin=nbin)[0])[0])
    r0 = float(first[-1])
    for r1 in (1.0, 0.98 * rout):
        for target in sorted({bin_of(r) for r in np.linspace(r0, r1, 400)})[1:]:
            lo, hi = r0, r1
            while True:
                mid = 0.5 * (lo + hi)
                if mid in (lo, hi):
                    break
                if bin_of(mid) < target:
                    lo = mid
                else:
                    hi = mid
            for side in (-1.0, 1.0):
                r = lo
                for _ in range(6):
                    records.append(np.append(first[:-1], r))
                    r = math.nextafter(r, side * 1e9)
    d = np.array(records)
    if many:
        d = np.concatenate([np.repeat(d[:1], 400, axis=0), d[1:]])
    d = d[:, rng.permutation(npair)] if npair > 1 else d
    t = np.zeros((len(d), nb), dtype=np.int32)
    got, ns = c.fp_histogram(nb, d, t, nbin=nbin)
    want, wns = o.fp_histogram(nb, d, t, nbin=nbin)
    assert len(d) > 200 and ns == wns
    assert np.array_equal(got, want)
