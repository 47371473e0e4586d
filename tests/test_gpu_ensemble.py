"""The persistent ensemble kernel at the edges of what it counts and of what a run may change."""
import numpy as np
import pytest

import steps_gb300 as S
from helpers import err_stats, rel_err
from steps_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def test_more_tasks_than_an_int(engine):
    """A long run of many small realisations: 5 tasks (one pair item, four of 32 particles) for each of 8,191
    realisations make 40,955 a stage, 2.15e9 in 52,501 stages. Realisation 0 is two particles of mass 1 at distance 1
    falling from rest; the leapfrog in FP64 is the answer, to the FP32 rounding of the force (6e-8, a few of them)."""
    steps, h = 52500, 1e-6
    assert 5 * 8191 * (steps + 1) >= 1 << 31
    xs = [np.array([[0.0, 0.0, 0.0], [1.0, 0.0, 0.0]])] + [np.zeros((1, 3))] * 8190
    sizes = [len(x) for x in xs]
    engine.batch_set(xs, [np.ones(n) for n in sizes], [np.full(n, 1e-3) for n in sizes])
    engine.batch_run(S.params(S.R3), S.MIXED, steps, h, graph=1)
    x, v, F = engine.batch_get(0)
    d, w = 1.0, 0.0  # separation and its rate: d'' = -2 / d^2
    a = -2.0
    for _ in range(steps):
        w += 0.5 * h * a
        d += h * w
        a = -2.0 / (d * d)
        w += 0.5 * h * a
    assert 1.0 - d > 0.002  # the motion that is looked at
    assert abs((1.0 - (x[1, 0] - x[0, 0])) / (1.0 - d) - 1.0) < 1e-6
    assert abs((v[1, 0] - v[0, 0]) / w - 1.0) < 1e-6
    assert abs(F[0, 0] / (-0.5 * a) - 1.0) < 1e-6


@pytest.mark.parametrize("graph", [1, 2])
def test_tuning_leaves_the_state(engine, graph):
    """The first run times candidate shapes on the registered data. An unsoftened particle's self pair is 0 * inf, so its
    force is NaN, in every path; nothing else may be: not its position or velocity, nor the others' forces."""
    sets = [W.r3_compactified(n, 300.0, seed=n, displace=True) for n in (300, 700)]
    sets[0].eps[5] = 0.0
    engine.batch_set([s.x for s in sets], [s.m for s in sets], [s.eps for s in sets])
    engine.batch_run(S.params(S.R3), S.MIXED, 0, 1e-3, graph=graph)
    for k, s in enumerate(sets):
        x, v, F = engine.batch_get(k)
        assert np.array_equal(x, s.x) and not v.any()
        good = np.ones(len(F), bool)
        good[5] = k != 0
        assert np.array_equal(np.isfinite(F).all(1), good)
        engine.set_particles(s.m, s.eps)
        assert err_stats(F[good], engine.forces(s.x, S.params(S.R3), S.FP64)[good])["p99"] < 1e-5


@pytest.mark.parametrize("graph", [1, 2])
def test_precision_guard_between_runs(engine, graph):
    """A captured run is captured again when the precision guard changes: its forces are those of a run that had to be
    captured under the new guard (one of another length came between), and of the old guard once that is back."""
    sets = [W.r3_compactified(n, 300.0, seed=n, displace=True) for n in (3000, 900)]
    p = S.params(S.R3)

    def run(guard, steps=0):
        engine.set_guard(guard)
        engine.batch_set([s.x for s in sets], [s.m for s in sets], [s.eps for s in sets])
        engine.batch_run(p, S.MIXED, steps, 1e-3, graph=graph)
        return np.concatenate([engine.batch_get(k)[2] for k in range(len(sets))])

    try:
        before, fine = run(30.0), run(2.0)
        run(2.0, steps=1)
        assert np.array_equal(fine, run(2.0))
        assert not np.array_equal(fine, before)
        assert np.array_equal(before, run(30.0))
    finally:
        engine.set_guard(30.0)


def test_errors_as_one_sided(engine):
    """FP32 sums over as few terms as in the packed one-sided kernel with tiles of 128, and so the same errors against
    FP64: 122,000 particles give the median to 0.3 % and the 99th percentile to 1 % (1 sigma)."""
    sets = [W.r3_compactified(n, 300.0, seed=n + k, displace=True) for n in (4736, 9000, 20000, 27000) for k in (1, 2)]
    p = S.params(S.R3)
    engine.batch_set([s.x for s in sets], [s.m for s in sets], [s.eps for s in sets])
    engine.batch_run(p, S.MIXED, 0, 1e-3, graph=1)
    pairwise, one = [], []
    engine.set_variant(1)
    engine.set_tuning(128, 1, 0)
    try:
        for k, s in enumerate(sets):
            engine.set_particles(s.m, s.eps)
            F64 = engine.forces(s.x, p, S.FP64)
            pairwise.append(rel_err(engine.batch_get(k)[2], F64))
            one.append(rel_err(engine.forces(s.x, p, S.MIXED), F64))
    finally:
        engine.set_variant(0)
        engine.set_tuning(128, 2, 0)
    a, b = (np.percentile(np.concatenate(e), [50, 99]) for e in (pairwise, one))
    assert a[0] < 1.02 * b[0] and a[1] < 1.04 * b[1], (a, b)


@pytest.mark.parametrize("split", [1, 6, 16, 40, 1000])
def test_every_plan(engine, split):
    """Each plan that the first run times (and a coarser and a finer one), whichever it would choose: realisations
    below, at and above one tile, of one and of several tiles to a group, and 0 and 2 steps."""
    sizes = (1, 2, 127, 128, 129, 257, 900, 5000, 20000)
    sets = [W.r3_compactified(max(n, 2), 300.0, seed=n, displace=True) for n in sizes]
    xs, ms, es = ([getattr(s, f)[:n] for s, n in zip(sets, sizes)] for f in ("x", "m", "eps"))
    p, h = S.params(S.R3), 1e-3
    for steps in (0, 2):
        engine.batch_set(xs, ms, es)
        engine.test_ensemble_plan(split)
        engine.batch_run(p, S.MIXED, steps, h, graph=1)
        got = [engine.batch_get(k) for k in range(len(sizes))]
        for k, (x, v, F) in enumerate(got):
            engine.set_particles(ms[k], es[k])
            F64 = engine.forces(x, p, S.FP64)
            if sizes[k] == 1:
                assert not F.any() and not v.any() and np.array_equal(x, xs[k])
                continue
            assert err_stats(F, F64)["p99"] < 1e-5, (sizes[k], steps)
            if steps == 0:
                assert np.array_equal(x, xs[k]) and not v.any()
                continue
            engine.upload_positions(xs[k])
            engine.upload_velocities(np.zeros_like(xs[k]))
            engine.kdk(p, S.FP64, steps, h)
            x64, v64, _ = engine.state()
            assert np.abs(x - x64).max() < 1e-9 * (1 + np.abs(x64).max()), sizes[k]
            assert err_stats(v, v64)["p99"] < 1e-5, sizes[k]
    engine.test_ensemble_plan(0)
    for bad in (-1, 1001):
        with pytest.raises(S.StepsError) as e:
            engine.test_ensemble_plan(bad)
        assert e.value.code == S.STEPS_E_ARG
