"""The per-kernel entry points (tri_kernel_*_f64, one per reference device
kernel) against the oracle's restatement of the same kernel, on the same
seeded state, through the C ABI with device buffers."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

_dp = C.POINTER(C.c_double)
_ip = C.POINTER(C.c_int32)


def _state():
    from triton_b200 import scenarios
    sc = scenarios.mixed(rows=37, cols=51, seed=13, open_boundaries=0, friction=True, duration=5.0)
    return sc


def _dev(torch, a, dtype=None):
    t = torch.from_numpy(np.ascontiguousarray(a)).cuda()
    return t


def _p(t):
    return C.c_void_p(t.data_ptr())


def _np(a):
    return np.ascontiguousarray(a, dtype=np.float64).reshape(-1)


def test_kernel_entry_points_match_oracle(oracle):
    import torch
    from triton_b200 import _abi
    L = _abi.lib()
    O = oracle.lib()
    for f in ("tor_compute_dt_and_sqrt", "tor_flux_x", "tor_flux_y", "tor_update_cells", "tor_update_runoff",
              "tor_compute_flow", "tor_open_boundaries", "tor_compute_extbc_values", "tor_wet_dry",
              "tor_copy_observation_points"):
        getattr(O, f).restype = None
    sc = _state()
    R, Cc = sc.rows, sc.cols
    N = R * Cc
    h, qx, qy, z, n2 = (_np(getattr(sc, k)) for k in ("h", "qx", "qy", "z", "n2"))
    cn, hx, dx = sc.courant, sc.hextra, sc.dx
    # --- compute_dt_and_sqrt + find_min_dt
    sq_o, dt_o = np.zeros(N), np.zeros(N)
    O.tor_compute_dt_and_sqrt(N, C.c_double(dx), qx.ctypes.data_as(_dp), qy.ctypes.data_as(_dp),
                              h.ctypes.data_as(_dp), sq_o.ctypes.data_as(_dp), dt_o.ctypes.data_as(_dp),
                              C.c_double(cn), C.c_double(hx))
    dh, dqx, dqy, dz, dn2 = (_dev(torch, a) for a in (h, qx, qy, z, n2))
    dsq, ddt = torch.zeros(N, dtype=torch.float64, device="cuda"), torch.zeros(N, dtype=torch.float64, device="cuda")
    _abi.check(L.tri_kernel_compute_dt_and_sqrt_f64(N, dx, _p(dqx), _p(dqy), _p(dh), _p(dsq), _p(ddt), cn, hx, None))
    torch.cuda.synchronize()
    assert np.array_equal(dsq.cpu().numpy(), sq_o)
    assert np.array_equal(ddt.cpu().numpy(), dt_o)
    dmin = torch.zeros(1, dtype=torch.float64, device="cuda")
    _abi.check(L.tri_kernel_find_min_dt_f64(N, _p(ddt), _p(dmin), None))
    torch.cuda.synchronize()
    m = O.tor_find_min_dt(N, dt_o.ctypes.data_as(_dp))
    assert dmin.item() == m
    dt = m
    # --- flux_x, flux_y (rhs arrays start from random garbage, as in the reference nothing clears them)
    rng = np.random.default_rng(0)
    rhs_o = [rng.standard_normal(N) for _ in range(6)]
    rhs_d = [_dev(torch, a.copy()) for a in rhs_o]
    args_o = [a.ctypes.data_as(_dp) for a in rhs_o]
    O.tor_flux_x(R, Cc, C.c_double(dx), C.c_double(dt), h.ctypes.data_as(_dp), qx.ctypes.data_as(_dp),
                 qy.ctypes.data_as(_dp), z.ctypes.data_as(_dp), sq_o.ctypes.data_as(_dp), *args_o, C.c_double(hx))
    O.tor_flux_y(R, Cc, C.c_double(dx), C.c_double(dt), h.ctypes.data_as(_dp), qx.ctypes.data_as(_dp),
                 qy.ctypes.data_as(_dp), z.ctypes.data_as(_dp), sq_o.ctypes.data_as(_dp), *args_o, C.c_double(hx))
    _abi.check(L.tri_kernel_flux_x_f64(N, R, Cc, dx, dt, _p(dh), _p(dqx), _p(dqy), _p(dz), _p(dsq),
                                       *[_p(t) for t in rhs_d], hx, None))
    _abi.check(L.tri_kernel_flux_y_f64(N, R, Cc, dx, dt, _p(dh), _p(dqx), _p(dqy), _p(dz), _p(dsq),
                                       *[_p(t) for t in rhs_d], hx, None))
    torch.cuda.synchronize()
    for a, t in zip(rhs_o, rhs_d):
        assert np.array_equal(t.cpu().numpy(), a)
    # --- update_cells (friction: cube root, tolerance)
    O.tor_update_cells(R, Cc, C.c_double(dt), h.ctypes.data_as(_dp), qx.ctypes.data_as(_dp), qy.ctypes.data_as(_dp),
                       n2.ctypes.data_as(_dp), *args_o, C.c_double(hx))
    _abi.check(L.tri_kernel_update_cells_f64(N, R, Cc, dt, _p(dh), _p(dqx), _p(dqy), _p(dz), _p(dn2),
                                             *[_p(t) for t in rhs_d], hx, None))
    torch.cuda.synchronize()
    for a, t in ((h, dh), (qx, dqx), (qy, dqy)):
        g = t.cpu().numpy()
        assert np.abs(g - a).max() <= 1e-12 * max(np.abs(a).max(), 1.0)
    # continue from identical states
    for a, t in ((h, dh), (qx, dqx), (qy, dqy)):
        t.copy_(torch.from_numpy(a))
    # --- runoff
    ro = sc.runoff
    zone = np.ascontiguousarray(ro["zone"].reshape(-1), dtype=np.int32)
    rates = _np(ro["rates"])
    nrows = ro["times"].size
    O.tor_update_runoff(R, Cc, C.c_double(dt), zone.ctypes.data_as(_ip), 2, nrows, rates.ctypes.data_as(_dp),
                        h.ctypes.data_as(_dp), qx.ctypes.data_as(_dp), qy.ctypes.data_as(_dp), C.c_double(hx))
    dzone, drates = _dev(torch, zone), _dev(torch, rates)
    _abi.check(L.tri_kernel_update_runoff_f64(N, R, Cc, dt, _p(dzone), 2, nrows, _p(drates), _p(dh), _p(dqx), _p(dqy),
                                              hx, None))
    # --- point sources (two share a cell)
    so = sc.sources
    cells = np.ascontiguousarray(so["cells"], dtype=np.int32)
    ht, hv = _np(so["times"]), _np(so["flows"])
    O.tor_compute_flow(cells.size, ht.ctypes.data_as(_dp), hv.ctypes.data_as(_dp), C.c_double(dx), C.c_double(dt),
                       C.c_double(3.0), 0, 1, h.ctypes.data_as(_dp), cells.ctypes.data_as(_ip))
    dcells, dht, dhv = _dev(torch, cells), _dev(torch, ht), _dev(torch, hv)
    _abi.check(L.tri_kernel_compute_flow_f64(cells.size, _p(dht), _p(dhv), dx, dt, 3.0, 0, 1, _p(dh), _p(dcells),
                                             None))
    # --- open boundaries (west/east then north/south)
    O.tor_open_boundaries(R, Cc, h.ctypes.data_as(_dp), qx.ctypes.data_as(_dp), qy.ctypes.data_as(_dp))
    _abi.check(L.tri_kernel_copy_info_to_exterior_boundaries_west_east_f64(2 * R, R, Cc, _p(dh), _p(dqx), _p(dqy),
                                                                           None))
    _abi.check(L.tri_kernel_copy_info_to_exterior_boundaries_north_south_f64(Cc, R, Cc, _p(dh), _p(dqx), _p(dqy), 0,
                                                                             1, None))
    torch.cuda.synchronize()
    for a, t in ((h, dh), (qx, dqx), (qy, dqy)):
        assert np.array_equal(t.cpu().numpy(), a)
    # --- external boundaries
    e = sc.extbc
    arrs = [np.ascontiguousarray(e[k], dtype=np.int32) for k in ("cells", "types", "start", "nrows")]
    v1, v2 = _np(e["var1"]), _np(e["var2"])
    O.tor_compute_extbc_values(arrs[0].size, R, Cc, C.c_double(dt), h.ctypes.data_as(_dp), qx.ctypes.data_as(_dp),
                               qy.ctypes.data_as(_dp), z.ctypes.data_as(_dp), n2.ctypes.data_as(_dp),
                               *[a.ctypes.data_as(_ip) for a in arrs], v1.ctypes.data_as(_dp),
                               v2.ctypes.data_as(_dp), C.c_double(7.0))
    darrs = [_dev(torch, a) for a in arrs]
    dv1, dv2 = _dev(torch, v1), _dev(torch, v2)
    _abi.check(L.tri_kernel_compute_extbc_values_f64(arrs[0].size, R, Cc, dt, _p(dh), _p(dqx), _p(dqy), _p(dz),
                                                     _p(dn2), *[_p(t) for t in darrs], _p(dv1), _p(dv2), 7.0, 0, 1,
                                                     None))
    torch.cuda.synchronize()
    for a, t in ((h, dh), (qx, dqx), (qy, dqy)):
        g = t.cpu().numpy()
        assert np.abs(g - a).max() <= 1e-12 * max(np.abs(a).max(), 1.0)
        t.copy_(torch.from_numpy(a))
    # --- wet_dry + max depth
    maxh = h.copy() * 0.5
    dmaxh = _dev(torch, maxh.copy())
    O.tor_wet_dry(R, Cc, h.ctypes.data_as(_dp), qx.ctypes.data_as(_dp), qy.ctypes.data_as(_dp), z.ctypes.data_as(_dp),
                  maxh.ctypes.data_as(_dp), C.c_double(hx))
    _abi.check(L.tri_kernel_wet_dry_f64(N, R, Cc, dt, _p(dh), _p(dqx), _p(dqy), _p(dz), _p(dmaxh), hx, 1, None))
    torch.cuda.synchronize()
    for a, t in ((qx, dqx), (qy, dqy), (maxh, dmaxh)):
        assert np.array_equal(t.cpu().numpy(), a)
    # --- observation gather
    obs = np.ascontiguousarray(sc.obs_cells, dtype=np.int32)
    out_o = np.zeros(obs.size)
    O.tor_copy_observation_points(obs.size, h.ctypes.data_as(_dp), out_o.ctypes.data_as(_dp), obs.ctypes.data_as(_ip))
    dobs, dout = _dev(torch, obs), torch.zeros(obs.size, dtype=torch.float64, device="cuda")
    _abi.check(L.tri_kernel_copy_observation_points_f64(obs.size, _p(dh), _p(dout), _p(dobs), None))
    torch.cuda.synchronize()
    assert np.array_equal(dout.cpu().numpy(), out_o)


@pytest.mark.parametrize("n", [1, 127, 128, 129, 1025, 9000])
@pytest.mark.parametrize("odd", [False, True])
def test_extbc_list_order_matches_oracle(oracle, n, odd):
    """Boundary cells listed several times with different types, in any order
    (each cell's items apply in list order), around the sizes of a block, of
    the scan's chunk and beyond the scan's limit; a list with a ghost cell in
    it is applied serially.  Types without a cube root: equal in every bit."""
    import torch
    from triton_b200 import _abi
    L, O = _abi.lib(), oracle.lib()
    O.tor_compute_extbc_values.restype = None
    R, Cc = 43, 61
    rng = np.random.default_rng(n)
    edge = [r * Cc + c for r in range(1, R - 1) for c in range(1, Cc - 1) if r in (1, R - 2) or c in (1, Cc - 2)]
    cells = rng.choice(np.array(edge, np.int32), n).astype(np.int32)
    if odd:
        cells[n // 2] = 1  # ghost (0, 1): its column has a western ghost
    types = rng.choice(np.array([0, 1, 3], np.int32), n).astype(np.int32)
    start = np.where(types == 1, 0, 4).astype(np.int32)
    nrows = np.where(types == 1, 4, 1).astype(np.int32)
    v1, v2 = np.array([0.0, 5.0, 9.0, 30.0, 0.7]), np.array([6.0, 7.0, 6.5, 6.5, 0.7])
    h = rng.random(R * Cc) * 2.0
    qx, qy = rng.standard_normal(R * Cc), rng.standard_normal(R * Cc)
    z, n2 = 5.0 + rng.random(R * Cc), np.full(R * Cc, 1e-3)
    dev = [_dev(torch, a.copy()) for a in (h, qx, qy, z, n2, cells, types, start, nrows, v1, v2)]
    O.tor_compute_extbc_values(n, R, Cc, C.c_double(0.1), *[a.ctypes.data_as(_dp) for a in (h, qx, qy, z, n2)],
                               *[a.ctypes.data_as(_ip) for a in (cells, types, start, nrows)],
                               v1.ctypes.data_as(_dp), v2.ctypes.data_as(_dp), C.c_double(7.0))
    _abi.check(L.tri_kernel_compute_extbc_values_f64(n, R, Cc, 0.1, *[_p(t) for t in dev], 7.0, 0, 1, None))
    torch.cuda.synchronize()
    for a, t in zip((h, qx, qy), dev):
        assert np.array_equal(t.cpu().numpy(), a)


@pytest.mark.parametrize("n", [1, 31, 32, 33, 100])
def test_flow_of_sources_in_shared_cells_matches_oracle(oracle, n):
    """Sources that share cells add up in source order, within a warp's 32
    sources and across them."""
    import torch
    from triton_b200 import _abi
    L, O = _abi.lib(), oracle.lib()
    O.tor_compute_flow.restype = None
    rng = np.random.default_rng(n)
    h = rng.random(50)
    pos = rng.choice(np.array([3, 17, 44], np.int32), n).astype(np.int32)
    ht, hv = np.array([0.0, 4.0, 9.0]), rng.random(3 * n)
    dh, dpos, dht, dhv = (_dev(torch, a.copy()) for a in (h, pos, ht, hv))
    O.tor_compute_flow(n, ht.ctypes.data_as(_dp), hv.ctypes.data_as(_dp), C.c_double(3.0), C.c_double(0.07),
                       C.c_double(3.0), 0, 1, h.ctypes.data_as(_dp), pos.ctypes.data_as(_ip))
    _abi.check(L.tri_kernel_compute_flow_f64(n, _p(dht), _p(dhv), 3.0, 0.07, 3.0, 0, 1, _p(dh), _p(dpos), None))
    torch.cuda.synchronize()
    assert np.array_equal(dh.cpu().numpy(), h)


def _flux_both(oracle, R, Cc, h, qx, qy, z, sq, hx, dx=3.0, dt=0.05):
    """flux_x then flux_y by the oracle and by the entries: two lists of six arrays."""
    import torch
    from triton_b200 import _abi
    L, O = _abi.lib(), oracle.lib()
    O.tor_flux_x.restype = O.tor_flux_y.restype = None
    want = [np.random.default_rng(k).standard_normal(R * Cc) for k in range(6)]
    got = [_dev(torch, a.copy()) for a in want]
    ins = [np.ascontiguousarray(a.reshape(-1)) for a in (h, qx, qy, z, sq)]
    dev = [_dev(torch, a) for a in ins]
    for name in ("x", "y"):
        getattr(O, "tor_flux_" + name)(R, Cc, C.c_double(dx), C.c_double(dt), *[a.ctypes.data_as(_dp) for a in ins],
                                       *[a.ctypes.data_as(_dp) for a in want], C.c_double(hx))
        _abi.check(getattr(L, f"tri_kernel_flux_{name}_f64")(R * Cc, R, Cc, dx, dt, *[_p(t) for t in dev],
                                                             *[_p(t) for t in got], hx, None))
    torch.cuda.synchronize()
    return want, [t.cpu().numpy() for t in got]


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
def test_flux_over_nonfinite_beds_matches_oracle(oracle, value):
    """Deep water over beds that are no number: the limiter's fmax and fmin
    replace the source term, so the contributions are finite."""
    rng = np.random.default_rng(2)
    R, Cc = 17, 40
    h = 2.0 + 0.2 * rng.random((R, Cc))
    z = 0.1 * rng.random((R, Cc))
    for r, c in ((0, 3), (5, 5), (5, 6), (6, 5), (16, 39)):
        z[r, c] = value
    zero = np.zeros((R, Cc))
    want, got = _flux_both(oracle, R, Cc, h, zero, zero, z, np.sqrt(h), 1e-3)
    for a, b in zip(want, got):
        assert np.isfinite(a).all() and np.array_equal(a, b)


@pytest.mark.parametrize("R,Cc", [(3, 3), (3, 9), (9, 3), (4, 4), (5, 7), (43, 61)])
def test_extbc_lists_of_any_cells_match_oracle(oracle, R, Cc):
    """Lists of cells of the whole grid, ghosts and corners among them, in any
    order and repeated; some cells write into others' ghosts."""
    import torch
    from triton_b200 import _abi
    L, O = _abi.lib(), oracle.lib()
    O.tor_compute_extbc_values.restype = None
    for n in (2, 5, 33, 700, 5000):
        rng = np.random.default_rng(100 * R + Cc + n)
        cells = rng.integers(0, R * Cc, n).astype(np.int32)
        types = rng.choice(np.array([0, 1, 3], np.int32), n).astype(np.int32)
        start, nrows = np.where(types == 1, 0, 4).astype(np.int32), np.where(types == 1, 4, 1).astype(np.int32)
        v1, v2 = np.array([0.0, 5.0, 9.0, 30.0, 0.7]), np.array([6.0, 7.0, 6.5, 6.5, 0.7])
        h, qx, qy = rng.random(R * Cc) * 2.0, rng.standard_normal(R * Cc), rng.standard_normal(R * Cc)
        z, n2 = 5.0 + rng.random(R * Cc), np.full(R * Cc, 1e-3)
        dev = [_dev(torch, a.copy()) for a in (h, qx, qy, z, n2, cells, types, start, nrows, v1, v2)]
        O.tor_compute_extbc_values(n, R, Cc, C.c_double(0.1), *[a.ctypes.data_as(_dp) for a in (h, qx, qy, z, n2)],
                                   *[a.ctypes.data_as(_ip) for a in (cells, types, start, nrows)],
                                   v1.ctypes.data_as(_dp), v2.ctypes.data_as(_dp), C.c_double(7.0))
        _abi.check(L.tri_kernel_compute_extbc_values_f64(n, R, Cc, 0.1, *[_p(t) for t in dev], 7.0, 0, 1, None))
        torch.cuda.synchronize()
        for a, t in zip((h, qx, qy), dev):
            assert np.array_equal(t.cpu().numpy(), a)


def test_extbc_lists_with_ghosts_or_repeats_stay_parallel():
    """A list of 8192 cells with a ghost in it, or with cells listed twice, takes
    no more than a few times a list of distinct interior cells (one thread for
    all of it took a hundred times as long, a thread's search for a cell's later
    items fifteen times)."""
    import torch
    from triton_b200 import _abi
    L, R, n = _abi.lib(), 2052, 8192
    edge = [r * R + c for r in (1, R - 2) for c in range(1, R - 1)] + [r * R + c for r in range(2, R - 2) for c in (1, R - 2)]
    edge = np.random.default_rng(1).permutation(np.array(edge, np.int32))
    f = [torch.rand(R * R, dtype=torch.float64, device="cuda") for _ in range(5)]
    types, zero = torch.full((n,), 3, dtype=torch.int32, device="cuda"), torch.zeros(n, dtype=torch.int32, device="cuda")
    one, v = torch.ones(n, dtype=torch.int32, device="cuda"), torch.full((1,), 0.3, dtype=torch.float64, device="cuda")
    us = {}
    for name, cells in (("plain", edge[:n]), ("ghost", np.append(edge[:n - 1], np.int32(1))), ("twice", np.tile(edge[:n // 2], 2))):
        t = _dev(torch, cells.astype(np.int32))
        best = 1e30
        for _ in range(5):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(10):
                _abi.check(L.tri_kernel_compute_extbc_values_f64(
                    n, R, R, 0.1, *[_p(x) for x in f], _p(t), _p(types), _p(zero), _p(one), _p(v), _p(v), 1.0, 0, 1,
                    C.c_void_p(torch.cuda.current_stream().cuda_stream)))
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b) * 100.0)
        us[name] = best
    assert us["ghost"] < 4 * us["plain"] and us["twice"] < 4 * us["plain"], us


_DEPTHS = [0.0, -0.0, 1e-310, 1e-95, 1e-12, 1e-3, 0.7, 0.9999999999999999, 3.0, 1e40]


@pytest.mark.parametrize("hx", [1e-3, 1e-40, 0.0])
def test_flux_of_values_past_the_straight_line_range_matches_oracle(oracle, hx):
    """Faces between depths of any size, at rest and with large discharges in
    ordinary depths; a threshold of zero with every cell wet."""
    rng = np.random.default_rng(3)
    R, Cc = 37, 53
    h = rng.choice(np.array(_DEPTHS if hx else _DEPTHS[3:]), (R, Cc))
    z = rng.random((R, Cc))
    big = rng.choice(np.array([0.0, 0.3, -2.0, 1e31, -1e35]), (R, Cc))
    qx = np.where((h > 1e-3) & (h < 4.0), big, 0.0)
    qy = np.where((h > 1e-3) & (h < 4.0), rng.permutation(big), 0.0)
    want, got = _flux_both(oracle, R, Cc, h, qx, qy, z, np.maximum(np.sqrt(h), 0.0), hx)
    for a, b in zip(want, got):
        assert np.isfinite(a).all() and np.array_equal(a, b)


@pytest.mark.parametrize("hx", [1e-3, 1e-40, 0.0])
def test_dt_of_values_past_the_straight_line_range_matches_oracle(oracle, hx):
    """Wave speeds of depths and discharges of any size, NaN and infinity among them."""
    import torch
    from triton_b200 import _abi
    L, O = _abi.lib(), oracle.lib()
    O.tor_compute_dt_and_sqrt.restype = None
    hs = np.array(_DEPTHS + [np.nan, np.inf, -1.0, 1e300, 5e-324])
    qs = np.array([0.0, -0.0, 5e-324, 1e-300, 0.3, -7.0, 1e31, 1e35, 1e300, np.nan, np.inf, -np.inf])
    h, qx, qy = (np.ascontiguousarray(a.reshape(-1)) for a in np.meshgrid(hs, qs, qs, indexing="ij"))
    n = h.size
    sq, dt = np.zeros(n), np.zeros(n)
    O.tor_compute_dt_and_sqrt(n, C.c_double(3.0), qx.ctypes.data_as(_dp), qy.ctypes.data_as(_dp), h.ctypes.data_as(_dp),
                              sq.ctypes.data_as(_dp), dt.ctypes.data_as(_dp), C.c_double(0.5), C.c_double(hx))
    dev = [_dev(torch, a) for a in (qx, qy, h)]
    dsq, ddt = torch.zeros(n, dtype=torch.float64, device="cuda"), torch.zeros(n, dtype=torch.float64, device="cuda")
    _abi.check(L.tri_kernel_compute_dt_and_sqrt_f64(n, 3.0, *[_p(t) for t in dev], _p(dsq), _p(ddt), 0.5, hx, None))
    torch.cuda.synchronize()
    assert np.array_equal(dsq.cpu().numpy(), sq, equal_nan=True)
    assert np.array_equal(ddt.cpu().numpy(), dt, equal_nan=True)
