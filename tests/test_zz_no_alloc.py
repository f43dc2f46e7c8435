"""tri_kernel_compute_extbc_values_noalloc_f64 (external-boundary cells with
the application order in a fixed device array instead of allocated scratch)
against tri_kernel_compute_extbc_values_f64 on the same device state.

The file is named to be collected last, so the no-alloc entry's first call on
the device (the address lookup of its fixed array) also runs after every
other test has used the library; the test passes alone and after the rest."""
import ctypes as C

import numpy as np
import pytest

from triton_b200 import _abi


def _p(t):
    return C.c_void_p(t.data_ptr())


def test_noalloc_rejects_lists_over_its_limit():
    # host-side check, before any CUDA call
    L = _abi.lib()
    n = _abi.NOALLOC_EXTBC_MAX_CELLS + 1
    rc = L.tri_kernel_compute_extbc_values_noalloc_f64(n, 10, 10, 0.1, *([None] * 11), 0.0, 0, 1, None)
    assert rc == _abi.TRI_E_INVALID
    assert b"fixed limit of 65536" in L.tri_last_error()


@pytest.mark.gpu
def test_noalloc_extbc_matches_allocating_entry():
    import torch
    from triton_b200 import scenarios
    L = _abi.lib()
    sc = scenarios.mixed(rows=37, cols=51, seed=13, open_boundaries=0, friction=True, duration=5.0)
    R, Cc = sc.rows, sc.cols
    dev = lambda a, dt=torch.float64: torch.as_tensor(np.ascontiguousarray(a), dtype=dt).reshape(-1).cuda()
    e = sc.extbc
    lists = [dev(e[k], torch.int32) for k in ("cells", "types", "start", "nrows")]
    dv1, dv2 = dev(e["var1"]), dev(e["var2"])
    dz, dn2 = dev(sc.z), dev(sc.n2)
    state = {}
    for arm in ("alloc", "noalloc"):
        state[arm] = [dev(getattr(sc, k)) for k in ("h", "qx", "qy")]
    entries = {"alloc": L.tri_kernel_compute_extbc_values_f64,
               "noalloc": L.tri_kernel_compute_extbc_values_noalloc_f64}

    def call(arm, cells, dt, simtime):
        n = cells[0].numel()
        h, qx, qy = state[arm]
        _abi.check(entries[arm](n, R, Cc, dt, _p(h), _p(qx), _p(qy), _p(dz), _p(dn2), *[_p(t) for t in cells],
                                _p(dv1), _p(dv2), simtime, 0, 1, None))

    def same(where):
        torch.cuda.synchronize()
        for name, a, b in zip(("h", "qx", "qy"), state["alloc"], state["noalloc"]):
            assert torch.equal(a, b), f"{where}: {name} differs in {int((a != b).sum())} cells"

    # two calls in a row with the same cell list
    for k, (dt, t) in enumerate(((0.05, 7.0), (0.04, 7.05))):
        for arm in ("alloc", "noalloc"):
            call(arm, lists, dt, t)
        same(f"call {k + 1}")
    # then another cell list (every second cell, reversed): the order is rebuilt
    sub = [t[::2].flip(0).contiguous() for t in lists]
    for arm in ("alloc", "noalloc"):
        call(arm, sub, 0.03, 7.09)
    same("call 3, other list")
    # and the first list again
    for arm in ("alloc", "noalloc"):
        call(arm, lists, 0.05, 7.12)
    same("call 4, first list again")


@pytest.mark.gpu
@pytest.mark.parametrize("entry", ["tri_kernel_compute_extbc_values_f64", "tri_kernel_compute_extbc_values_noalloc_f64"])
def test_long_lists_keep_and_rebuild_their_order(oracle, entry):
    """Lists above 8192 cells, whose order the host finds and keeps (in allocated
    scratch, or in the no-alloc entry's fixed array): a list twice in a row, a
    longer one, one of the same length with other cells, the first again, against
    the oracle.  Types without a cube root: every bit."""
    import torch
    L, O = _abi.lib(), oracle.lib()
    O.tor_compute_extbc_values.restype = None
    R, Cc = 43, 61
    rng = np.random.default_rng(71)
    edge = np.array([r * Cc + c for r in range(1, R - 1) for c in range(1, Cc - 1)
                     if r in (1, R - 2) or c in (1, Cc - 2)], np.int32)

    def lists(n):
        types = rng.choice(np.array([0, 1, 3], np.int32), n).astype(np.int32)
        return (rng.choice(edge, n).astype(np.int32), types, np.where(types == 1, 0, 4).astype(np.int32),
                np.where(types == 1, 4, 1).astype(np.int32))

    v1, v2 = np.array([0.0, 5.0, 9.0, 30.0, 0.7]), np.array([6.0, 7.0, 6.5, 6.5, 0.7])
    state = [rng.random(R * Cc) * 2.0, rng.standard_normal(R * Cc), rng.standard_normal(R * Cc)]
    z, n2 = 5.0 + rng.random(R * Cc), np.full(R * Cc, 1e-3)
    dev = [torch.from_numpy(a.copy()).cuda() for a in state + [z, n2, v1, v2]]
    ptr = lambda a: a.ctypes.data_as(C.c_void_p)
    first, longer, other = lists(9000), lists(12000), lists(9000)
    for k, cells in enumerate((first, first, longer, other, first)):
        n, t = cells[0].size, 7.0 + 0.5 * k
        O.tor_compute_extbc_values(n, R, Cc, C.c_double(0.1), *[ptr(a) for a in state + [z, n2]],
                                   *[ptr(a) for a in cells], ptr(v1), ptr(v2), C.c_double(t))
        dc = [torch.from_numpy(a).cuda() for a in cells]
        _abi.check(getattr(L, entry)(n, R, Cc, 0.1, *[_p(x) for x in dev[:5]], *[_p(x) for x in dc], _p(dev[5]),
                                     _p(dev[6]), t, 0, 1, None))
        torch.cuda.synchronize()
        for name, a, b in zip(("h", "qx", "qy"), state, dev):
            assert np.array_equal(b.cpu().numpy(), a), f"call {k + 1}: {name}"
