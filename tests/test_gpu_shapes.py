"""The one-sided kernel shape and j split that are chosen when the caller set none, at the sizes where the choice
changes, against the FP64 kernels."""
import pytest

import steps_gb300 as S
from helpers import err_stats
from steps_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture
def fresh(engine):
    """The engine with no shape or variant chosen."""
    engine.shutdown()
    yield S.Engine(0)
    engine.set_tuning(128, 2, 0)
    engine.set_variant(0)


# (n, first, count): one particle, one tile, below and above 3e7, 1.5e8 and 8e9 pairs, short ranges against many particles
RANGES = [(1, 0, 1), (64, 0, 63), (65, 1, 64), (5001, 0, 4990), (5011, 0, 5005), (100003, 5, 1), (100003, 50000, 33),
          (120001, 20000, 66000), (120001, 0, 67500), (5475, 0, 5475), (5479, 0, 5479),
          (12247, 0, 12247), (12248, 0, 12248)]


@pytest.mark.parametrize("n,lo,count", RANGES)
def test_r3(fresh, n, lo, count):
    ps = W.r3_compactified(n, 480.0, seed=n, displace=True)
    fresh.set_particles(ps.m, ps.eps)
    p = S.params(S.R3, cosmology=1, comoving=1, mius=1e-3)
    F = fresh.forces(ps.x, p, S.MIXED, lo, lo + count - 1)
    k = min(count, 500)
    assert err_stats(F[-k:], fresh.forces(ps.x, p, S.FP64, lo + count - k, lo + count - 1))["p99"] < 1e-5


@pytest.mark.parametrize("n", [1, 2, 31, 512, 513, 1024, 1025, 2049, 4097, 8192, 8193, 16385, 32767, 32768, 32769])
def test_ordering_sizes(fresh, n):
    """Sets of up to 32,768 particles are ordered by one cluster of 1 to 8 blocks, 2, 4 or 8 particles a thread; with
    coincident particles, one far outlier and (in y) all at one value."""
    ps = W.r3_compactified(max(n, 2), 480.0, seed=n, displace=True)
    x = ps.x[:n].copy()
    x[:, 1] = 3.0
    x[n // 2:n // 2 + 5] = x[0]
    x[-1, 0] += 1e7
    fresh.set_particles(ps.m[:n], ps.eps[:n])
    p = S.params(S.R3)
    F = fresh.forces(x, p, S.MIXED)
    k = min(n, 400)
    st = err_stats(F[:k], fresh.forces(x, p, S.FP64, 0, k - 1))
    assert st["p99"] < 1e-5 or n == 1, st


@pytest.mark.parametrize("n", [32769, 34816, 34817, 67584, 67585, 262144, 262145])
def test_radix_ordering_sizes(fresh, n):
    """Larger sets: whole and partial sort blocks, one and two rounds of the digit scan, 4 and 5 passes; with
    coincident particles, one far outlier and (in y) all at one value."""
    ps = W.r3_compactified(n, 480.0, seed=n, displace=True)
    x = ps.x.copy()
    x[:, 1] = 3.0
    x[n // 2:n // 2 + 5] = x[0]
    x[-1, 0] += 1e7
    fresh.set_particles(ps.m, ps.eps)
    p = S.params(S.R3)
    F = fresh.forces(x, p, S.MIXED)
    for lo in (0, n // 2 - 200, n - 400):
        st = err_stats(F[lo:lo + 400], fresh.forces(x, p, S.FP64, lo, lo + 399))
        assert st["p99"] < 1e-5, (n, lo, st)


@pytest.mark.parametrize("kind", ["t3", "tab0", "tab2", "img"])
@pytest.mark.parametrize("n,lo,count", [(63, 0, 63), (4095, 0, 4095), (40000, 100, 24000), (40000, 100, 26000)])
def test_periodic(fresh, kind, n, lo, count):
    """Wide stencils change shape at 1e9 pairs; below n = 4,096 full ranges are one-sided."""
    if kind == "t3":
        ps, p = W.t3_clumpy(n, 100.0, 3), S.params(S.T3, is_periodic=2, L=100.0, rsim=50.0, ewald_order=4)
        fresh.build_table_t3(31, 100.0, 0.02, 2.0, 0.3, 3.0, 6.0)
    else:
        ps = W.s1r2_cylindrical(n, 200.0, 600.0, 2)
        p = S.params(S.S1R2, is_periodic=2, L=200.0, rsim=600.0, s1r2_images=int(kind == "img"),
                     ewald_order=int(kind[-1]) if kind != "img" else 4)
        fresh.build_table_s1r2(432, 64, 1350.0, 200.0, 0.787875 / 200.0, 4, 10)
    fresh.set_particles(ps.m, ps.eps)
    F = fresh.forces(ps.x, p, S.MIXED, lo, lo + count - 1)
    k = min(count, 300)
    assert err_stats(F[-k:], fresh.forces(ps.x, p, S.FP64, lo + count - k, lo + count - 1))["p99"] < 1e-5


@pytest.mark.parametrize("count", [9890, 9910])
def test_tricubic_line(fresh, count):
    """Tricubic ranges change shape at 1e8 pairs."""
    n = 10100  # 1e8 pairs lie between the two counts
    ps, p = W.t3_clumpy(n, 100.0, 3), S.params(S.T3, is_periodic=2, L=100.0, rsim=50.0, ewald_order=4)
    fresh.build_table_t3(31, 100.0, 0.02, 2.0, 0.3, 3.0, 6.0)
    fresh.set_particles(ps.m, ps.eps)
    lo = n - count
    F = fresh.forces(ps.x, p, S.MIXED, lo, n - 1)
    assert err_stats(F[-300:], fresh.forces(ps.x, p, S.FP64, n - 300, n - 1))["p99"] < 1e-5
    fresh.set_tuning(64 if count * n < 1e8 else 256, 1, 0)
    assert (F == fresh.forces(ps.x, p, S.MIXED, lo, n - 1)).all()


@pytest.mark.parametrize("kind", ["r3", "t3"])
def test_autotune_replaces_a_set_shape(fresh, kind):
    """After steps_gpu_autotune an earlier explicit choice no longer counts, for the ranges of a call whose all-particle
    form is not timed either."""
    n = 24000
    if kind == "t3":
        ps, p = W.t3_clumpy(n, 100.0, 3), S.params(S.T3, is_periodic=2, L=100.0, rsim=50.0, ewald_order=2)
        fresh.build_table_t3(31, 100.0, 0.02, 2.0, 0.3, 3.0, 6.0)
    else:
        ps, p = W.r3_compactified(n, 480.0, seed=4, displace=True), S.params(S.R3)
    fresh.set_particles(ps.m, ps.eps)
    want = fresh.forces(ps.x, p, S.MIXED), fresh.forces(ps.x, p, S.MIXED, 100, 9000)
    fresh.set_variant(0)
    fresh.set_tuning(64, 4 if kind == "r3" else 2, 3)  # T^3 has no 64 x 4
    assert not (want[0] == fresh.forces(ps.x, p, S.MIXED)).all()
    assert not (want[1] == fresh.forces(ps.x, p, S.MIXED, 100, 9000)).all()
    fresh.upload_positions(ps.x)
    fresh.autotune(p)
    assert (want[0] == fresh.forces(ps.x, p, S.MIXED)).all()
    assert (want[1] == fresh.forces(ps.x, p, S.MIXED, 100, 9000)).all()
