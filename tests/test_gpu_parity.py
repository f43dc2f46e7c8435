"""Parity of the GPU domain path (C ABI, fused sm_100a kernels) with the CPU
oracle on the same seeded inputs.

The plain FP64 form must equal the oracle bit for bit where no cube root is
involved (CUDA's cbrt and glibc's may differ in the last bit), and otherwise
stay within 1e-9 of each field's scale with identical wet/dry masks."""
import numpy as np
import pytest

from tests._harness import run_lockstep

pytestmark = pytest.mark.gpu


def test_dambreak_bit_exact():
    from triton_b200 import scenarios
    sc = scenarios.dambreak(n=96, dx=1.0, radius=20.0, depth=5.0, duration=3.0)
    sc.print_interval = 1.0
    steps, nev = run_lockstep(sc, exact=True)
    assert steps > 20 and nev >= 3


def test_dambreak_odd_shape():
    from triton_b200 import scenarios
    sc = scenarios.dambreak(n=70, dx=0.5, radius=9.0, depth=2.0, duration=2.0)
    # make it rectangular and odd: drop columns
    for k in ("z", "h", "qx", "qy", "n2"):
        setattr(sc, k, getattr(sc, k)[:, :47].copy())
    sc.z[:, -1] = 1e6
    sc.h[:, -1] = 0.0
    run_lockstep(sc, exact=True)


def test_thacker_small_bit_exact():
    from triton_b200 import scenarios
    sc = scenarios.thacker(n=128, dx=64.0, periods=0.05)
    sc.print_interval = sc.sim_duration / 2
    steps, _ = run_lockstep(sc, exact=True)
    assert steps > 10


@pytest.mark.parametrize("open_b", [0, 1])
def test_mixed_no_cbrt_bit_exact(open_b):
    from triton_b200 import scenarios
    sc = scenarios.mixed(rows=41, cols=57, seed=11 + open_b, open_boundaries=open_b, friction=False,
                         with_extbc=False, duration=12.0)
    steps, nev = run_lockstep(sc, exact=True)
    assert steps > 10 and nev > 3


@pytest.mark.parametrize("seed", [3, 4])
def test_mixed_all_forcing(seed):
    from triton_b200 import scenarios
    sc = scenarios.mixed(rows=33, cols=61, seed=seed, open_boundaries=0, friction=True, duration=15.0)
    steps, nev = run_lockstep(sc, exact=False)
    assert steps > 10


def test_mixed_open_boundaries_with_extbc():
    from triton_b200 import scenarios
    sc = scenarios.mixed(rows=29, cols=31, seed=21, open_boundaries=1, friction=True, duration=10.0)
    run_lockstep(sc, exact=False)


def test_wide_grid_multiple_strips():
    # more columns than one strip and more rows than one row block
    from triton_b200 import scenarios
    sc = scenarios.mixed(rows=150, cols=300, seed=5, friction=False, with_extbc=False, duration=4.0)
    run_lockstep(sc, exact=True, check_every_event=False)


def test_exact_division_selftest():
    """The kernels divide by dx and dt through a correctly rounded reciprocal
    and one Markstein correction; the quotient must equal IEEE a/b in every
    bit over the operand ranges the step produces."""
    import ctypes as C
    from triton_b200 import _abi
    bad = C.c_int64(-1)
    _abi.check(_abi.lib().tri_selftest_division(50_000_000, 12345, C.byref(bad)))
    assert bad.value == 0


def test_autotune_keeps_state_and_parity():
    from tests._harness import compare_fields, oracle_from_scenario, oracle_bookkeeping, domain_bookkeeping
    from triton_b200 import scenarios
    sc = scenarios.dambreak(n=120, dx=1.0, radius=25.0, depth=4.0, duration=2.0)
    o = oracle_from_scenario(sc)
    d = sc.to_domain()
    try:
        t = d.autotune(trial_steps=4)
        assert t["candidates"] >= 3 and t["ms_per_step"] > 0
        assert d.get_clock().it_count == 0
        while True:
            n1, e1 = o.advance(10 ** 6)
            n2, e2 = d.advance(10 ** 6)
            assert (n1, e1) == (n2, e2)
            compare_fields(o, d, True, sc.hextra)
            oracle_bookkeeping(o, e1)
            domain_bookkeeping(d, e2)
            if e1 & 1:
                break
    finally:
        d.close()


@pytest.mark.parametrize("shape", [(40, 61), (33, 30)])
@pytest.mark.parametrize("value", [0.0, 1e-310, 1e-250, 1e95])
def test_extreme_depths_bit_exact(value, shape):
    """Depths outside the range of the flux tile's straight-line arithmetic
    (2^-300 .. 2^300; 0 is inside) in some tiles of an ordinary wet case, on
    tile edges too: those tiles take the guarded forms and must still equal
    the oracle bit for bit."""
    from triton_b200 import scenarios
    rows, cols = shape
    sc = scenarios.mixed(rows=rows, cols=cols, seed=31, friction=False, with_extbc=False, with_sources=False,
                         with_runoff=False, duration=4.0)
    for r, c in ((1, 1), (8, 30), (9, 31 if cols > 31 else 5), (rows, cols)):
        sc.h[r, c] = value
        sc.qx[r, c] = sc.qy[r, c] = 0.0
    steps, _ = run_lockstep(sc, exact=True, max_events=1, chunk=6)
    assert 0 < steps <= 6  # an observation event may come first


@pytest.mark.parametrize("rows,cols,open_b", [(5, 31, 0), (33, 61, 1), (64, 30, 1), (40, 92, 0)])
def test_tile_heights_match_oracle(rows, cols, open_b):
    """Every tile height gives the oracle's bits: tiles of one row, heights that
    leave a remainder, one tile over the whole height; strips of 30 columns with
    1, 30 and 32 columns left; sources (two in one cell), runoff, zero-gradient
    edges."""
    from tests._harness import compare_fields, domain_bookkeeping, oracle_bookkeeping, oracle_from_scenario
    from triton_b200 import scenarios
    for variant, rb in ((0, 1), (1, 3), (2, 7), (0, 32), (0, 100)):
        sc = scenarios.mixed(rows=rows, cols=cols, seed=41, open_boundaries=open_b, friction=False, with_extbc=False,
                             duration=2.0)
        o, d = oracle_from_scenario(sc), sc.to_domain()
        try:
            d.set_shape(variant, rb)
            for _ in range(4):
                n1, e1 = o.advance(10 ** 6)
                n2, e2 = d.advance(10 ** 6)
                assert (n1, e1) == (n2, e2)
                assert d.get_clock().simtime == o.s.simtime
                compare_fields(o, d, True, sc.hextra, where=f"height {rb}: ")
                oracle_bookkeeping(o, e1)
                domain_bookkeeping(d, e2)
        finally:
            d.close()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_tile_heights_agree_with_boundary_cells(precision):
    """External boundary cells of every type, friction, arrival tracking: the
    default height, tiles of one row and tall tiles give the same bits (a
    corner's ghosts belong to its tile at any height)."""
    from triton_b200 import scenarios
    got = []
    for rb in (0, 1, 4, 40):
        sc = scenarios.mixed(rows=37, cols=65, seed=43, friction=True, duration=5.0)
        sc.z[1:-1, 1:-1] += 700.0  # FP32: bed levels far from their bases' zero
        d = sc.to_domain(precision)
        try:
            if rb:
                d.set_shape(0, rb)
            d.track_arrival(0.3)
            d.set_clock(sim_duration=1e300, print_interval=1e300, time_series=0, it_print=0)
            assert d.advance(61)[0] == 61
            got.append([d.download(f) for f in ("h", "qx", "qy", "maxh")] + [d.arrival(), np.array(d.get_clock().simtime)])
        finally:
            d.close()
    for other in got[1:]:
        for a, b in zip(got[0], other):
            assert np.array_equal(a, b)


@pytest.mark.parametrize("rb", [1 << 30, (1 << 31) - 1])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_any_tile_height_computes_every_tile(precision, rb):
    """Heights far above the grid's: a tile is taken in as many parts as its
    rows need (2^27 parts of 8 rows in each of 32 strips are 2^32, no part at
    all in 32 bits), alone and in a batch; the height set is the one reported."""
    from triton_b200 import _abi, scenarios
    from triton_b200.batch import Batch
    import ctypes as C
    got = []
    for mode in ("default", "domain", "batch"):
        sc = scenarios.mixed(rows=20, cols=960, seed=47, duration=5.0)
        d = sc.to_domain(precision)
        try:
            d.set_clock(sim_duration=1e300, print_interval=1e300, time_series=0, it_print=0)
            if mode == "batch":
                with Batch([d]) as b:
                    b.set_shape(0, rb)
                    assert b.advance(9).steps == 9
            else:
                if mode == "domain":
                    d.set_shape(0, rb)
                    t = _abi.Tuning()
                    _abi.check(_abi.lib().tri_domain_get_tuning(d._h, C.byref(t)))
                    assert t.rows_per_tile == rb
                assert d.advance(9)[0] == 9
            got.append([d.download(f) for f in ("h", "qx", "qy", "maxh")] + [np.array(d.get_clock().simtime)])
        finally:
            d.close()
    for other in got[1:]:
        for a, b in zip(got[0], other):
            assert np.array_equal(a, b)


def test_bed_without_a_level_under_water_matches_oracle():
    """Bed cells without a level (NaN) under water: the limiter replaces the
    source term that is not a number, as the oracle's fmax does, so the first
    step stays finite and equal in every bit."""
    from tests._harness import compare_fields, oracle_from_scenario
    from triton_b200 import scenarios
    sc = scenarios.mixed(rows=40, cols=61, seed=5, friction=False, with_extbc=False, with_sources=False,
                         with_runoff=False, duration=1e3)
    rng = np.random.default_rng(5)
    sc.h[1:-1, 1:-1] = 2.0 + 0.2 * rng.random((40, 61))
    sc.qx[:], sc.qy[:] = 0.0, 0.0
    sc.z[1:-1, 1:-1] = 0.1 * rng.random((40, 61))
    for r, c in ((3, 3), (9, 31), (9, 32), (10, 30), (20, 30), (33, 7)):
        sc.z[r, c] = np.nan
    o, d = oracle_from_scenario(sc), sc.to_domain()
    try:
        assert o.advance(1) == d.advance(1) == (1, 0)
        assert np.isfinite(o.grid("h")).all() and np.isfinite(o.grid("qx")).all()
        compare_fields(o, d, True, sc.hextra)
        assert d.get_clock().simtime == o.s.simtime
    finally:
        d.close()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_cells_without_a_depth_stay_apart(precision):
    """A block of cells without a depth (NaN) inside dry land: its faces have
    no water on either side and add nothing, so its discharges stay zero and
    nothing spreads, as in the oracle (FP64: every bit)."""
    from tests._harness import compare_fields, oracle_from_scenario
    from triton_b200 import scenarios
    sc = scenarios.mixed(rows=40, cols=61, seed=5, friction=False, with_extbc=False, with_sources=False,
                         with_runoff=False, duration=1e3)
    for f in (sc.h, sc.qx, sc.qy):
        f[:14, :34] = 0.0
    sc.h[2:7, 3:30] = np.nan
    d = sc.to_domain(precision)
    try:
        assert d.advance(3) == (3, 0)
        if precision == "fp64":
            o = oracle_from_scenario(sc)
            assert o.advance(3) == (3, 0)
            compare_fields(o, d, True, sc.hextra)
        assert np.array_equal(np.isnan(d.download("h")), np.isnan(sc.h))
        for f in ("qx", "qy"):
            assert not d.download(f)[2:7, 3:30].any()
    finally:
        d.close()


@pytest.mark.parametrize("hextra", [0.0, 1e-300, 1e-40])
def test_any_depth_threshold_matches_oracle(hextra):
    """Thresholds down to zero (all wet there: a dry cell's velocity is 0/0),
    whose films and their velocities have any size."""
    from triton_b200 import scenarios
    sc = scenarios.mixed(rows=40, cols=61, seed=53, friction=False, with_extbc=False, open_boundaries=1, duration=4.0)
    sc.hextra = hextra
    if hextra == 0.0:
        sc.h += 0.25
    else:
        sc.h[9:13, 25:35] = hextra * 1.5  # at rest: a discharge there would leave the range of doubles
        sc.qx[9:13, 25:35] = sc.qy[9:13, 25:35] = 0.0
    steps, _ = run_lockstep(sc, exact=True, max_events=2, chunk=8)
    assert steps > 1


def _flux_us(sc):
    """Time of a flux launch of an FP64 domain, the shortest of three runs of 16 steps."""
    d = sc.to_domain()
    best = 1e30
    try:
        d.set_clock(sim_duration=1e300, print_interval=1e300, time_series=0, it_print=0)
        d.advance(8)
        for _ in range(3):
            d.set_timing(True)
            d.advance(16)
            ms, n, _, _ = d.get_timing()
            best = min(best, 1e3 * ms / n)
        d.set_timing(False)
    finally:
        d.close()
    return best


def _wet_square(n=700):
    from triton_b200 import scenarios
    sc = scenarios.mixed(rows=n, cols=n, seed=59, with_extbc=False, with_sources=False, duration=1e3)
    rng = np.random.default_rng(59)
    sc.h[1:-1, 1:-1] = 1.0 + 0.2 * rng.random((n, n))
    sc.qx[:], sc.qy[:] = 0.0, 0.0
    return sc


def test_small_depth_threshold_takes_the_straight_line_form():
    """With a threshold below 2^-100 no tile is computed twice (2.5 times the
    launch when each was)."""
    sc = _wet_square()
    usual = _flux_us(sc)
    sc.hextra = 1e-40
    assert _flux_us(sc) < 1.5 * usual


def test_depths_of_minus_zero_are_dry_land():
    """Depths of -0.0 equal the oracle's run bit for bit, and a tile with
    them is computed once (1.5 times the launch when it was twice)."""
    from triton_b200 import scenarios
    sc = scenarios.mixed(rows=40, cols=61, seed=61, friction=False, duration=4.0)
    sc.extbc = None
    sc.h[sc.h == 0.0] = -0.0
    run_lockstep(sc, exact=True, max_events=2, chunk=6)
    times = []
    for dry in (0.0, -0.0):
        sc = _wet_square()
        sc.runoff = None
        sc.h[np.random.default_rng(67).random(sc.h.shape) < 0.5] = dry
        times.append(_flux_us(sc))
    assert times[1] < 1.25 * times[0], times


def test_autotune_tries_the_default_shape():
    """The default height of this grid (3 rows) is not one of the heights that
    every budget is tried at; the default is tried beside them, alone and in a
    batch.  A default among them is not tried twice."""
    from triton_b200 import scenarios
    from triton_b200.batch import Batch
    for cols, tried in ((1050, 31), (200, 30)):
        sc = scenarios.mixed(rows=200, cols=cols, seed=73, with_extbc=False, duration=1e3)
        d = sc.to_domain()
        try:
            assert d.autotune(2)["candidates"] == tried
            with Batch([d]) as b:
                assert b.autotune(2)["candidates"] == tried
        finally:
            d.close()


def _odd_cells(sc, depth, discharge):
    rows, cols = sc.rows - 2, sc.cols - 2
    for r, c in ((1, 1), (8, 30), (9, 31 if cols > 31 else 5), (rows, cols)):
        sc.h[r, c] = depth
        sc.qx[r, c], sc.qy[r, c] = discharge, -discharge
    return sc


@pytest.mark.parametrize("depth,discharge,hextra,steps", [(1e40, 0.0, 1e-3, 6), (1e-95, 0.0, 1e-100, 4),
                                                          (1.0, 1e35, 1e-3, 2), (1.0, 1e31, 1e-3, 4)])
def test_values_past_the_straight_line_range_match_oracle(depth, discharge, hextra, steps):
    """Depths above 2^100, wet ones below 2^-300 and discharges above 2^100 on
    tile edges: those tiles, and the wave speeds of such cells, take the guarded
    forms, bit for bit, alone and as a member of a batch."""
    from tests._harness import compare_fields, oracle_from_scenario
    from triton_b200 import scenarios
    from triton_b200.batch import Batch
    for batch in (False, True):
        sc = scenarios.mixed(rows=40, cols=61, seed=31, friction=False, with_extbc=False, with_sources=False,
                             with_runoff=False, duration=1e3)
        sc.hextra = hextra
        _odd_cells(sc, depth, discharge)
        o, d = oracle_from_scenario(sc), sc.to_domain()
        try:
            o.advance(steps)
            if batch:
                with Batch([d]) as b:
                    b.set_shape(0, 8)
                    b.advance(steps)
            else:
                d.advance(steps)
            assert all(np.isfinite(o.grid(f)).all() for f in ("h", "qx", "qy"))
            assert d.get_clock().simtime == o.s.simtime
            compare_fields(o, d, True, hextra)
        finally:
            d.close()


def _uniform_flow(h, qx, qy, n2, hextra):
    """A flat channel in uniform flow: one step changes its inner cells by
    friction alone."""
    from triton_b200 import scenarios
    sc = scenarios.mixed(rows=40, cols=45, seed=1, with_extbc=False, with_sources=False, with_runoff=False, duration=1e3)
    sc.hextra = hextra
    sc.h[1:-1, 1:-1], sc.qx[1:-1, 1:-1], sc.qy[1:-1, 1:-1] = h, qx, qy
    sc.z[1:-1, 1:-1], sc.n2[:] = 0.0, n2
    return sc


_FLOWS = [(1.0, 0.3, 0.2, 1e-3, 1e-3), (1.0, 0.3, 0.0, 1e-3, 1e-3), (1.0, 0.3, 1e-70, 1e-3, 1e-3),
          (1.0, 0.3, 1e-250, 1e-3, 1e-3), (1.0, 0.3, 0.2, 1e19, 1e-3), (1.0, 1e-11, 0.0, 1e-3, 1e-3),
          (1.0, 3e-13, 0.0, 1e-3, 1e-3), (1e-40, 2e-12, 1e-100, 1e-3, 1e-45), (1.0, 0.3, 0.2, 1e-11, 1e-3)]


@pytest.mark.parametrize("h,qx,qy,n2,hextra", _FLOWS)
def test_friction_over_its_range_matches_oracle(h, qx, qy, n2, hextra):
    """Friction terms of any size, transverse discharges that have decayed, both
    sides of the thresholds.  Tolerance: the cube root's last bits move the
    friction term t by a few ulps, and the reference's -(m - m*s)/(2t) loses
    1/t of its digits: 8 ulps times 1 + 1/t."""
    from tests._harness import oracle_from_scenario
    sc = _uniform_flow(h, qx, qy, n2, hextra)
    o, d = oracle_from_scenario(sc), sc.to_domain()
    try:
        assert o.advance(1) == d.advance(1) == (1, 0)
        inner = (slice(6, -6), slice(6, -6))
        t = o.s.global_dt * 9.81 * n2 * np.hypot(qx, qy) / (h * h * np.cbrt(h))
        for f in ("qx", "qy"):
            a, w = d.download(f)[inner], o.grid(f)[inner]
            assert np.abs(a - w).max() <= 8 * 2.0 ** -52 * (1 + 1 / t) * np.abs(w).max() + 5e-324, f
        assert np.array_equal(d.download("h")[inner], o.grid("h")[inner])
    finally:
        d.close()


@pytest.mark.parametrize("h,qx,qy,n2,hextra", _FLOWS)
def test_friction_of_guarded_tiles_has_the_same_bits(h, qx, qy, n2, hextra):
    """The same cells in a tile that holds a cell out of range (too far away to
    reach them in a step) and in one that does not."""
    got = []
    for odd in (False, True):
        sc = _uniform_flow(h, qx, qy, n2, hextra)
        sc.h[1, 1], sc.qx[1, 1], sc.qy[1, 1] = 1e-310 if odd else 0.0, 0.0, 0.0
        d = sc.to_domain()
        try:
            d.set_shape(0, 40)
            d.set_clock(time_increment_fixed=1, time_step=1e-40 if h < 1 else 0.05)
            assert d.advance(1)[0] == 1
            got.append([d.download(f)[8:-1, 8:-1] for f in ("h", "qx", "qy")])
        finally:
            d.close()
    for a, b in zip(*got):
        assert np.array_equal(a, b)
