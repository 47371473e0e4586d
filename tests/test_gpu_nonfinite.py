"""Positions that are NaN or infinite: every index made from them stays inside its table (a call returns NaN where the
position matters, as the arithmetic has it, and the next call is right)."""
import math

import numpy as np
import pytest

import steps_gb300 as S
from steps_gb300 import workloads as W

pytestmark = pytest.mark.gpu

L3, LZ = 100.0, 200.0


@pytest.fixture
def fresh(engine):
    """The engine with no shape or variant chosen."""
    engine.shutdown()
    yield S.Engine(0)
    engine.set_tuning(128, 2, 0)
    engine.set_variant(0)


def system(eng, kind, n):
    if kind == "r3":
        return W.r3_compactified(n, 480.0, 1, True), S.params(S.R3)
    if kind.startswith("t3"):
        eng.build_table_t3(17, L3, 2.0 / L3, 2.0, 5.0 * 2.0 * math.pi / L3, 3.0, 6.0)
        return W.t3_clumpy(n, L3, 1), S.params(S.T3, is_periodic=2, L=L3, rsim=L3 / 2, ewald_order=int(kind[2:]))
    if kind.startswith("table"):
        eng.build_table_s1r2(200, 64, 2.25 * 600.0, LZ, 0.787875 / LZ, 4, 10)
    return W.s1r2_cylindrical(n, LZ, 600.0, 1), S.params(S.S1R2, is_periodic=2, L=LZ, rsim=600.0,
                                                       s1r2_images=int(kind == "images"),
                                                       ewald_order=int(kind[5:]) if kind.startswith("table") else 4)


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf, 1e300])
@pytest.mark.parametrize("kind", ["r3", "t32", "t34", "images", "table0", "table2", "table4"])
def test_position(fresh, kind, value):
    """One coordinate of one particle, along each axis; both precisions, all particles (one-sided and each pair once)
    and a range."""
    for n in (700, 4200):
        ps, p = system(fresh, kind, n)
        fresh.set_particles(ps.m, ps.eps)
        for precision in (S.MIXED, S.FP64):
            before = fresh.forces(ps.x, p, precision)
            for axis in range(3):
                x = ps.x.copy()
                x[n // 3, axis] = value
                F = fresh.forces(x, p, precision)
                part = fresh.forces(x, p, precision, n // 3 - 5, n // 3 + 5)
                if not np.isfinite(value) and not (kind == "images" and axis == 2):  # there, no image is inside the cut
                    assert np.isnan(F[n // 3]).any() and np.isnan(part[5]).any()
            assert np.array_equal(before, fresh.forces(ps.x, p, precision))


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf, 1e300])
def test_cylindrical_background(fresh, value):
    """The radial-force table of a comoving S^1 x R^2 run is read at the particle's own radius."""
    n = 700
    ps = W.s1r2_cylindrical(n, LZ, 600.0, 1)
    fresh.build_radial_table(1000, 600.0, LZ, 1000)
    fresh.set_particles(ps.m, ps.eps)
    p = S.params(S.S1R2, is_periodic=2, L=LZ, rsim=600.0, s1r2_images=1, cosmology=1, comoving=1, mius=1e-3)
    for precision in (S.MIXED, S.FP64):
        before = fresh.forces(ps.x, p, precision)
        for axis in (0, 1):
            x = ps.x.copy()
            x[n // 3, axis] = value
            F = fresh.forces(x, p, precision)
            if not np.isfinite(value):
                assert np.isnan(F[n // 3]).any()
        assert np.array_equal(before, fresh.forces(ps.x, p, precision))
