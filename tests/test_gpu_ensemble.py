"""The persistent ensemble kernel at the edges of what it counts and of what a run may change."""
import numpy as np
import pytest

import steps_gb300 as S

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
