"""The pairwise kernels at the sizes of the workloads, where groups hold many rows and every chunk is in use, against
the FP64 kernels on three samples of i particles: an engine on which no shape or variant was chosen runs them for all
particles."""
import math

import numpy as np
import pytest

import steps_gb300 as S
from helpers import err_stats
from steps_gb300 import workloads as W

pytestmark = pytest.mark.gpu

SAMPLE = 1024


@pytest.fixture
def fresh(engine):
    """The engine with no shape or variant chosen."""
    engine.shutdown()
    yield S.Engine(0)
    engine.set_tuning(128, 2, 0)
    engine.set_variant(0)


def check(eng, ps, p):
    eng.set_particles(ps.m, ps.eps)
    F = eng.forces(ps.x, p, S.MIXED)
    assert np.isfinite(F).all()
    for lo in (0, ps.n // 2 - 7, ps.n - SAMPLE):
        st = err_stats(F[lo:lo + SAMPLE], eng.forces(ps.x, p, S.FP64, lo, lo + SAMPLE - 1))
        assert st["p99"] < 1e-5, (lo, st)


@pytest.mark.parametrize("n", [1 << 18, 700001, 1 << 20])
def test_r3(fresh, n):
    check(fresh, W.r3_compactified(n, 1000.0, seed=1, displace=True), S.params(S.R3, cosmology=1, comoving=1, mius=1e-3))


@pytest.mark.parametrize("order", [2, 4])
def test_t3(fresh, order):
    fresh.build_table_t3(63, 100.0, 2.0 / 100.0, 2.0, 5.0 * 2.0 * math.pi / 100.0, 3.0, 6.0)
    ps = W.workload("cfg3") if order == 2 else W.t3_clumpy(200001, 100.0, seed=3)
    check(fresh, ps, S.params(S.T3, is_periodic=2, L=100.0, rsim=50.0, ewald_order=order))


@pytest.mark.parametrize("order", [2, 4])
def test_s1r2_table(fresh, order):
    fresh.build_table_s1r2(864, 128, 2.25 * 600.0, 200.0, 0.787875 / 200.0, 4, 10)
    ps = W.s1r2_cylindrical((1 << 20) if order == 2 else 400001, 200.0, 600.0, seed=2)
    check(fresh, ps, S.params(S.S1R2, is_periodic=2, L=200.0, rsim=600.0, s1r2_images=0, ewald_order=order))


def test_s1r2_images(fresh):
    ps = W.s1r2_cylindrical(1 << 20, 200.0, 600.0, seed=2)
    check(fresh, ps, S.params(S.S1R2, is_periodic=2, L=200.0, rsim=600.0, s1r2_images=1))
