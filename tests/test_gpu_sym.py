"""The pairwise kernels (each pair of particles evaluated once, added to both)
against the FP64 kernels, at the edges of tiles, rows, row widths and groups."""
import numpy as np
import pytest

import steps_gb300 as S
from helpers import err_stats
from steps_gb300 import workloads as W

pytestmark = pytest.mark.gpu

MIXED_P99 = 1e-5


@pytest.fixture
def fresh(engine):
    """The engine with no shape or variant chosen."""
    engine.shutdown()
    eng = S.Engine(0)
    yield eng
    eng.set_tuning(128, 2, 0)
    eng.set_variant(0)


@pytest.mark.parametrize("n", [16384, 16385, 16511, 20001, 65535, 65536, 65600, 70001])
def test_r3_sizes(fresh, n):
    """Taken from n = 16,384 on; wider rows from 65,536 on, where groups hold several rows from 65,537 on."""
    ps = W.r3_compactified(n, 480.0, seed=n, displace=True)
    fresh.set_particles(ps.m, ps.eps)
    p = S.params(S.R3, cosmology=1, comoving=1, mius=1e-3)
    F = fresh.forces(ps.x, p, S.MIXED)
    for lo in (0, max(0, n - 3000)):
        hi = min(n, lo + 3000) - 1
        st = err_stats(F[lo:hi + 1], fresh.forces(ps.x, p, S.FP64, lo, hi))
        assert st["p99"] < MIXED_P99, (n, lo, st)
    assert np.array_equal(F, fresh.forces(ps.x, p, S.MIXED))  # fixed summation order


def test_r3_softened_and_coincident(fresh):
    """Pairs inside the spline, a coincident pair, and unsoftened particles beside
    padding (their self pair is 0 * inf in the FP64 kernel, as in the reference)."""
    rng = np.random.default_rng(5)
    x = rng.normal(0, 0.5, (16500, 3))
    x[1] = x[0]
    eps = np.full(16500, 0.1)
    eps[16400:] = 0.0
    m = rng.uniform(0.5, 2.0, 16500)
    fresh.set_particles(m, eps)
    F = fresh.forces(x, S.params(S.R3), S.MIXED)
    F64 = fresh.forces(x, S.params(S.R3), S.FP64)
    ok = np.isfinite(F64).all(1)
    assert ok[:16400].all() and np.array_equal(np.isfinite(F).all(1), ok)
    assert err_stats(F[ok], F64[ok])["p99"] < MIXED_P99


@pytest.mark.parametrize("scale", [1e-9, 1e9, 1e13])
def test_r3_units(fresh, scale):
    """Lengths far from 1: r^-3 itself leaves the FP32 range at 1e13, its products with the masses do not; at 1e-9
    those products overflow in the softened core. Nothing the one-sided kernel represents is lost."""
    ps = W.r3_compactified(16500, 480.0, seed=3, displace=True)
    m = ps.m * 1e10
    fresh.set_particles(m, ps.eps * scale)
    p = S.params(S.R3)
    F64 = fresh.forces(ps.x * scale, p, S.FP64)
    F = fresh.forces(ps.x * scale, p, S.MIXED)
    fresh.set_variant(1)
    one = fresh.forces(ps.x * scale, p, S.MIXED)
    ok = np.isfinite(one).all(1)
    assert np.isfinite(F).all(1)[ok].all()
    if ok.any():
        assert err_stats(F[ok], F64[ok])["p99"] < MIXED_P99
    assert ok.any() or scale < 1


def test_r3_kdk_and_choice(fresh):
    """The leapfrog on it, and an explicit pair loop switching it off: the same forces to rounding."""
    ps = W.r3_compactified(17000, 480.0, seed=11, displace=True)
    p = S.params(S.R3)
    out = []
    for variant in (None, 1):
        if variant is not None:
            fresh.set_variant(variant)
        fresh.set_particles(ps.m, ps.eps)
        fresh.upload_positions(ps.x)
        fresh.upload_velocities(np.zeros_like(ps.x))
        fresh.kdk(p, S.MIXED, 3, 1e-3)
        out.append(fresh.state())
    assert err_stats(out[0][2], out[1][2])["p99"] < MIXED_P99
    assert np.abs(out[0][0] - out[1][0]).max() < 1e-6
