"""The pairwise kernels (each pair of particles evaluated once, added to both)
against the FP64 kernels, at the edges of tiles, rows, row widths and groups."""
import math
import time

import numpy as np
import pytest

import steps_gb300 as S
from helpers import err_stats, rel_err
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


@pytest.mark.parametrize("n", [16384, 16385, 16511, 19999, 20000, 20001, 39999, 40000, 65600, 70001, 99999, 100000, 100353])
def test_r3_sizes(fresh, n):
    """Taken from n = 20,000 on; groups of several rows from 32,769 on, wider rows from 100,000 on."""
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
    x = rng.normal(0, 0.5, (20500, 3))
    x[1] = x[0]
    eps = np.full(20500, 0.1)
    eps[20400:] = 0.0
    m = rng.uniform(0.5, 2.0, 20500)
    fresh.set_particles(m, eps)
    F = fresh.forces(x, S.params(S.R3), S.MIXED)
    F64 = fresh.forces(x, S.params(S.R3), S.FP64)
    ok = np.isfinite(F64).all(1)
    assert ok[:20400].all() and np.array_equal(np.isfinite(F).all(1), ok)
    assert err_stats(F[ok], F64[ok])["p99"] < MIXED_P99


@pytest.mark.parametrize("scale", [1e-9, 1e9, 1e13])
def test_r3_units(fresh, scale):
    """Lengths far from 1: r^-3 itself leaves the FP32 range at 1e13, its products with the masses do not; at 1e-9
    those products overflow in the softened core. Nothing the one-sided kernel represents is lost."""
    ps = W.r3_compactified(20500, 480.0, seed=3, displace=True)
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
    ps = W.r3_compactified(21000, 480.0, seed=11, displace=True)
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


# ---- periodic topologies ------------------------------------------------------

L3, LZ = 100.0, 200.0


def periodic(eng, kind, n, seed=1):
    """A workload set and parameters; the table, if the kind has one, is built."""
    if kind.startswith("t3"):
        ps = W.t3_clumpy(n, L3, seed)
        order = int(kind[2:])
        if order:
            eng.build_table_t3(31, L3, 2.0 / L3, 2.0, 5.0 * 2.0 * math.pi / L3, 3.0, 6.0)
        return ps, S.params(S.T3, is_periodic=2 if order else 1, L=L3, rsim=L3 / 2, ewald_order=order or 2)
    ps = W.s1r2_cylindrical(n, LZ, 600.0, seed)
    if kind == "s1tab2" or kind == "s1tab4":
        eng.build_table_s1r2(432, 64, 2.25 * 600.0, LZ, 0.787875 / LZ, 4, 10)
        return ps, S.params(S.S1R2, is_periodic=2, L=LZ, rsim=600.0, s1r2_images=0, ewald_order=int(kind[-1]))
    return ps, S.params(S.S1R2, is_periodic=int(kind[2:]), L=LZ, rsim=600.0, s1r2_images=1)


KINDS = ["t30", "t32", "t34", "s11", "s12", "s115", "s1tab2", "s1tab4"]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n", [4096, 4127, 8192, 8193, 16385, 33000])
def test_periodic_sizes(fresh, kind, n):
    """Taken from n = 4,096 on; groups are one block up to 8,192, two up to 16,384, whole tiles above."""
    ps, p = periodic(fresh, kind, n)
    fresh.set_particles(ps.m, ps.eps)
    F = fresh.forces(ps.x, p, S.MIXED)
    for lo in (0, n - 700):
        st = err_stats(F[lo:lo + 700], fresh.forces(ps.x, p, S.FP64, lo, lo + 699))
        assert st["p99"] < MIXED_P99, (kind, n, lo, st)
    assert np.array_equal(F, fresh.forces(ps.x, p, S.MIXED))


@pytest.mark.parametrize("ng", [5, 31, 129, 145])
@pytest.mark.parametrize("n", [1500, 4500])
def test_t3_brick_records(fresh, ng, n):
    """Trilinear records in bricks: grids of 1 and 3 (mod 4) cells, halo of 16 cells and wider; one-sided and
    pairwise, and particles over the whole box, so that cells at the edges of the haloed table are read."""
    ps = W.t3_clumpy(n, L3, 5)
    fresh.build_table_t3(ng, L3, 2.0 / L3, 2.0, 5.0 * 2.0 * math.pi / L3, 3.0, 6.0)
    p = S.params(S.T3, is_periodic=2, L=L3, rsim=L3 / 2, ewald_order=2)
    fresh.set_particles(ps.m, ps.eps)
    st = err_stats(fresh.forces(ps.x, p, S.MIXED), fresh.forces(ps.x, p, S.FP64))
    assert st["p99"] < MIXED_P99, (ng, n, st)


@pytest.mark.parametrize("kind", KINDS)
def test_periodic_hard_decisions(fresh, kind):
    """Pairs within a few FP32 ulps of half a period along each axis and of the image cut: the image is the FP64
    kernel's. (Pairs at half a period to the last FP64 bits, below the 48 bits that mixed positions hold, may fall
    either way in every mixed kernel: they are computed beside the others and not compared.)"""
    n = 6000
    ps, p = periodic(fresh, kind, n, seed=7)
    rng = np.random.default_rng(3)
    x = ps.x.copy()
    period = L3 if kind.startswith("t3") else LZ
    axes = (0, 1, 2) if kind.startswith("t3") else (2,)
    dist = [period / 2] + ([2.6 * LZ % LZ] if kind == "s12" else [])
    a, b = np.arange(0, 2000, 2), np.arange(1, 2000, 2)
    for k, (i, j) in enumerate(zip(a, b)):
        ax, d = axes[k % len(axes)], dist[k // 3 % len(dist)]
        x[j] = x[i] + rng.normal(0.0, 0.5, 3)
        x[j, ax] = x[i, ax] + d * (1.0 + (k % 7 - 3) * 2.0 ** -23)
        x[j] = x[j] if not kind.startswith("t3") else x[j] % period
        x[j, 2] %= period
    fresh.set_particles(ps.m, ps.eps)
    F = fresh.forces(x, p, S.MIXED)
    resolved = np.repeat(np.arange(1000) % 7 != 3, 2)
    st = err_stats(F[:2000][resolved], fresh.forces(x, p, S.FP64, 0, 1999)[resolved])
    assert st["p99"] < MIXED_P99, st
    assert st["max"] < 1e-3, st  # a flipped image moves a particle's force by per cents


@pytest.mark.parametrize("topology", ["t32", "s1tab2"])
def test_tables_that_are_not_odd(fresh, topology):
    """A table without the symmetry of an Ewald correction is used as given (by the one-sided kernels)."""
    n = 5000
    ps, p = periodic(fresh, topology, n)
    rng = np.random.default_rng(2)
    if topology == "t32":
        fresh.set_table_t3(rng.normal(0.0, 1e-4, 3 * 31 ** 3), 31)
    else:
        fresh.set_table_s1r2(rng.normal(0.0, 1e-6, 2 * 432 * 64), 432, 64)
    fresh.set_particles(ps.m, ps.eps)
    F = fresh.forces(ps.x, p, S.MIXED)
    fresh.set_tuning(64, 1, 0)  # the shape of one-sided periodic calls of this size
    assert np.array_equal(F, fresh.forces(ps.x, p, S.MIXED))


@pytest.mark.parametrize("precision", [S.MIXED, S.FP64])
@pytest.mark.parametrize("kind,entry", [("t32", 0), ("t32", 1), ("t34", 0), ("t34", 2), ("s1tab2", 0), ("s1tab2", 1)])
def test_tables_with_a_nan(fresh, kind, entry, precision):
    """One NaN in one component: only the particles whose own stencils read it get NaN, as one-sided."""
    n = 4500
    ps, p = periodic(fresh, kind, n)
    if kind.startswith("t3"):
        table = fresh.get_table_t3(31)
        table[3 * (31 * 31 * 9 + 31 * 14 + 20) + entry] = np.nan
        fresh.set_table_t3(table, 31)
    else:
        table = fresh.get_table_s1r2(432, 64)
        table[2 * (100 * 64 + 40) + entry] = np.nan
        fresh.set_table_s1r2(table, 432, 64)
    fresh.set_particles(ps.m, ps.eps)
    F = fresh.forces(ps.x, p, precision)
    half = np.concatenate([fresh.forces(ps.x, p, precision, 0, n // 2), fresh.forces(ps.x, p, precision, n // 2 + 1, n - 1)])
    bad = np.isnan(half)
    assert bad.any() and not bad.all()
    assert np.array_equal(np.isnan(F), bad)


@pytest.mark.parametrize("ng", [127, 255])
def test_first_call_after_a_table(fresh, ng):
    """The first call with a new table looks whether it is odd: one pass over it (50 and 400 MB, 10 and 60 us at the
    memory's rate) and one wait for the answer, so 0.5 ms more than a later call at most."""
    ps = W.t3_clumpy(1000, L3, 1)
    fresh.build_table_t3(ng, L3, 2.0 / L3, 2.0, 5.0 * 2.0 * math.pi / L3, 3.0, 6.0)
    table = fresh.get_table_t3(ng)
    p = S.params(S.T3, is_periodic=2, L=L3, rsim=L3 / 2, ewald_order=2)
    fresh.set_particles(ps.m, ps.eps)

    def call():
        t0 = time.perf_counter()
        fresh.forces(ps.x, p, S.FP64)
        return time.perf_counter() - t0

    first = []
    for _ in range(4):
        fresh.set_table_t3(table, ng)
        first.append(call())
    assert min(first) - min(call() for _ in range(4)) < 0.5e-3


# ---- FP64 -----------------------------------------------------------------------


@pytest.mark.parametrize("kind", ["r3", "t30", "t32", "t34", "s11", "s12", "s1tab2"])
@pytest.mark.parametrize("n", [511, 512, 543, 2000, 8193])
def test_fp64_sizes(fresh, kind, n):
    """All particles (each pair once, from n = 512 on) against the two halves (one-sided): the difference is the order
    of the sums, 1e-16 times a few. Groups hold two rows from 8,193 on."""
    if kind == "r3":
        ps, p = W.r3_compactified(n, 480.0, seed=n, displace=True), S.params(S.R3, cosmology=1, comoving=1, mius=1e-3)
    else:
        ps, p = periodic(fresh, kind, n)
    fresh.set_particles(ps.m, ps.eps)
    F = fresh.forces(ps.x, p, S.FP64)
    half = np.concatenate([fresh.forces(ps.x, p, S.FP64, 0, n // 2), fresh.forces(ps.x, p, S.FP64, n // 2 + 1, n - 1)])
    assert rel_err(F, half).max() < 1e-11
    assert np.median(rel_err(F, half)) < 1e-14
    assert np.array_equal(F, fresh.forces(ps.x, p, S.FP64))


def test_fp64_softened_and_far_units(fresh, port):
    """Pairs inside and at the edge of the spline, a coincident pair, and lengths where r^2 leaves the FP32 range."""
    import pyoracle as O
    from helpers import port_params
    rng = np.random.default_rng(5)
    x = rng.normal(0, 0.05, (600, 3))
    x[1] = x[0]
    x[3] = x[2] + np.array([0.2, 0, 0])
    m, eps = rng.uniform(0.5, 2.0, 600), np.full(600, 0.1)
    for scale in (1.0, 1e-12, 1e15):
        fresh.set_particles(m, eps * scale)
        F = fresh.forces(x * scale, S.params(S.R3), S.FP64)
        Fo = port.forces(port.system(0, m, eps * scale, port_params(O)), x * scale)
        assert rel_err(F, Fo).max() < 1e-11, scale


@pytest.mark.parametrize("entry", ["forces", "ranges", "noalloc"])
@pytest.mark.parametrize("scale", [1e-21, 1e-18, 3e18, 1e22])
def test_fp64_outside_the_fp32_range(fresh, port, scale, entry):
    """Lengths where r^2 is far below or above what FP32 holds (1.2e-38 to 3.4e38), or partly so; one pair in a hundred
    or so is softened."""
    import ctypes as C
    import pyoracle as O
    from helpers import port_params
    rng = np.random.default_rng(6)
    n = 600
    x = rng.normal(0, 1.0, (n, 3)) * scale
    m, eps = rng.uniform(0.5, 2.0, n), np.full(n, 0.1 * scale)
    p = S.params(S.R3)
    fresh.set_particles(m, eps)
    if entry == "forces":
        F = fresh.forces(x, p, S.FP64)
    elif entry == "ranges":
        F = np.concatenate([fresh.forces(x, p, S.FP64, 0, 299), fresh.forces(x, p, S.FP64, 300, n - 1)])
    else:
        torch = pytest.importorskip("torch")
        dx, dm, de = (torch.from_numpy(a).to("cuda") for a in (x, m, eps))
        dF = torch.empty((n, 3), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        fn = fresh.lib.steps_gpu_forces_fp64_noalloc
        fn.argtypes = [C.POINTER(S.Params), C.c_void_p, C.c_void_p, C.c_void_p, C.c_int, C.c_void_p, C.c_int, C.c_int,
                       C.c_void_p]
        assert fn(C.byref(p), dx.data_ptr(), dm.data_ptr(), de.data_ptr(), n, dF.data_ptr(), 0, n - 1, None) == S.STEPS_OK
        torch.cuda.synchronize()
        F = dF.cpu().numpy()
    Fo = port.forces(port.system(0, m, eps, port_params(O)), x)
    # FP64 sums of 600 terms: about 600 roundings of 1.1e-16 of the sum of magnitudes, which cancels to 1e-2 at worst
    assert rel_err(F, Fo).max() < 1e-11


# ---- device memory ----------------------------------------------------------------


@pytest.mark.parametrize("precision", [S.MIXED, S.FP64])
@pytest.mark.parametrize("kind", ["r3", "s12"])
def test_partial_sums_that_do_not_fit(fresh, kind, precision):
    """Where the pairwise kernel's partial sums do not fit in device memory the call runs the one-sided kernel, with its
    launches only (no attempt first) and its result; with the memory back it is pairwise again."""
    torch = pytest.importorskip("torch")
    n = 100000 if precision == S.MIXED else 30000
    ps, p = (W.r3_compactified(n, 480.0, seed=2, displace=True), S.params(S.R3)) if kind == "r3" else periodic(fresh, kind, n)

    def call(eng):
        before = eng.launch_count()
        F = eng.forces(ps.x, p, precision)
        return F, eng.launch_count() - before

    fresh.set_particles(ps.m, ps.eps)
    if precision == S.MIXED:  # the one-sided shape of this size
        if kind == "r3":
            fresh.set_variant(1)
        fresh.set_tuning(*((128, 2, 0) if kind == "r3" else (64, 1, 0)))
        one, launches = call(fresh)
    else:
        one = np.concatenate([fresh.forces(ps.x, p, precision, 0, 0), fresh.forces(ps.x, p, precision, 1, n - 1)])
        launches = 3
    fresh.shutdown()
    eng = S.Engine(0)
    eng.set_particles(ps.m[:4000], ps.eps[:4000])
    eng.forces(ps.x[:4000], p, precision)
    eng.set_particles(ps.m, ps.eps)
    torch.cuda.init()
    # the slabs: 24 bytes for each particle, at least 128 + 128 of them on average
    room = 24 * n * 150
    hold = torch.empty(torch.cuda.mem_get_info()[0] - room, dtype=torch.uint8, device="cuda")
    try:
        got = [call(eng) for _ in range(3)]
    finally:
        del hold
        torch.cuda.empty_cache()
    for F, count in got[1:]:  # the first call allocates what else it needs
        if precision == S.MIXED:
            assert np.array_equal(F, one)
        else:
            assert rel_err(F, one).max() < 1e-11
        assert count == launches
    F, count = call(eng)
    assert not np.array_equal(F, got[0][0])
    assert rel_err(F, one).max() < (1e-3 if precision == S.MIXED else 1e-11)
