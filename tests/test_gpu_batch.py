"""Batched ensembles: every member of a tri_batch must end exactly where the
same domain run alone ends (same fields bit for bit, same step count and
simulated time), whatever the mix of member sizes and forcing.  The solo
path is itself checked against the oracle by the parity tests."""
from __future__ import annotations

import numpy as np
import pytest

from triton_b200 import scenarios
from triton_b200.batch import Batch

pytestmark = pytest.mark.gpu


def _members():
    ms = scenarios.ensemble(members=6, seed=11, side_min=40, side_max=160, duration=600.0, rain_range=(50, 200))
    for i, sc in enumerate(ms):
        sc.print_interval = 150.0 + 50.0 * i  # uneven print events
        sc.it_print = 37 + i
    mx = scenarios.mixed(rows=37, cols=53, seed=5)
    mx.name = "mixed"
    # open edges (zero-gradient ghosts, kernels.h:437-512) with sources and runoff
    op = scenarios.mixed(rows=29, cols=44, seed=8, open_boundaries=1, with_extbc=False)
    op.name = "open"
    return ms + [mx, op]


def _solo(sc, precision):
    d = sc.to_domain(precision)
    try:
        d.run()
        c = d.get_clock()
        return {f: d.download(f) for f in ("h", "qx", "qy", "maxh")}, c.it_count, c.simtime
    finally:
        d.close()


@pytest.mark.parametrize("single_launch", [False, True], ids=["graphs", "single_launch"])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_batch_members_equal_solo_runs(precision, single_launch):
    """Both launch modes: one launch per kernel type and step (CUDA graphs),
    and one persistent launch per chunk of steps whose blocks take work items
    with per-member dependencies."""
    scs = _members()
    solo = [_solo(sc, precision) for sc in scs]
    doms = [sc.to_domain(precision) for sc in scs]
    try:
        with Batch(doms) as b:
            b.set_mode(single_launch)
            steps, updates = b.run()
        assert steps > 0 and updates > 0
        for sc, d, (fields, it, t) in zip(scs, doms, solo):
            c = d.get_clock()
            assert c.it_count == it, f"{sc.name}: {c.it_count} steps batched, {it} alone"
            assert c.simtime == t, f"{sc.name}: simtime {c.simtime!r} batched, {t!r} alone"
            for f, ref in fields.items():
                got = d.download(f)
                bad = got != ref
                assert not bad.any(), f"{sc.name}: {f} differs in {int(bad.sum())} cells"
    finally:
        for d in doms:
            d.close()


def test_batch_autotune_keeps_members():
    scs = _members()[:4]
    doms = [sc.to_domain("fp64") for sc in scs]
    try:
        before = [(d.download("h"), d.get_clock().simtime) for d in doms]
        with Batch(doms) as b:
            t = b.autotune(3)
            assert t["candidates"] >= 1 and t["ms_per_step"] > 0
            for d, (h, st) in zip(doms, before):
                assert np.array_equal(d.download("h"), h)
                assert d.get_clock().simtime == st
            b.run()
        solo = [_solo(sc, "fp64") for sc in scs]
        for d, (fields, it, _) in zip(doms, solo):
            assert d.get_clock().it_count == it
            assert np.array_equal(d.download("h"), fields["h"])
    finally:
        for d in doms:
            d.close()


def test_batch_rejects_bad_members():
    from triton_b200 import TriError
    sc = scenarios.dambreak(n=32, duration=0.5)
    a = sc.to_domain("fp64")
    b = sc.to_domain("fp32")
    try:
        with pytest.raises(TriError):
            Batch([a, b])
        with pytest.raises(TriError):
            Batch([a, a])
    finally:
        a.close()
        b.close()


@pytest.mark.parametrize("precision,small", [("fp64", 760), ("fp32", 1200)])
def test_a_large_member_among_many_small_ones_keeps_its_blocks(precision, small):
    """More members than the post kernel has resident blocks: a large one is not
    left to one block (the step took ten times the parts' own steps)."""
    import torch
    from triton_b200.domain import Domain

    def flat(rows, cols):
        d = Domain(rows, cols, 1.0, 0.5, 1e-3, 0, precision)
        d.upload("h", 1.0 + 0.1 * np.random.default_rng(rows).random((rows, cols)))
        d.set_clock(sim_duration=1e300, print_interval=1e300, it_print=0)
        return d

    def step_us(members):
        with Batch(members) as b:
            b.launch(8)
            b.wait()
            best = 1e30
            for _ in range(3):
                e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                torch.cuda.synchronize()
                e0.record()
                b.launch(32)
                b.wait()
                e1.record()
                torch.cuda.synchronize()
                best = min(best, e0.elapsed_time(e1) / 32 * 1e3)
            return best

    large, others = flat(1026, 1026), [flat(18, 20) for _ in range(small)]
    try:
        alone, rest, both = step_us([large]), step_us(others), step_us([large] + others)
        assert both < 2.0 * (alone + rest), (alone, rest, both)
    finally:
        for d in [large] + others:
            d.close()


_SOLO = {}


def _advanced(precision, steps):
    """Members whose tiles fill more than one round of the flux kernel's warps at
    6 rows and of the post kernel's at one row, and each one's fields after
    `steps` steps alone at its default shape."""
    if precision not in _SOLO:
        scs = _members()[4:] + scenarios.ensemble(members=2, seed=12, side_min=690, side_max=730, duration=600.0,
                                                  rain_range=(50, 200))
        got = []
        for sc in scs:
            d = sc.to_domain(precision)
            d.set_clock(sim_duration=1e300, print_interval=1e300, time_series=0, it_print=0)
            assert d.advance(steps)[0] == steps
            got.append([d.download(f) for f in ("h", "qx", "qy", "maxh")] + [np.array(d.get_clock().simtime)])
            d.close()
        _SOLO[precision] = scs, got
    return _SOLO[precision]


@pytest.mark.parametrize("variant,rb", [(0, 1), (1, 6), (2, 12), (0, 32), (1, 100)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_batch_tile_heights_equal_solo_runs(precision, variant, rb):
    """Heights that divide the members' rows and that leave short last rows,
    whole tiles and the last ones in parts, several post tiles a warp."""
    scs, solo = _advanced(precision, 21)
    doms = [sc.to_domain(precision) for sc in scs]
    try:
        for d in doms:
            d.set_clock(sim_duration=1e300, print_interval=1e300, time_series=0, it_print=0)
        with Batch(doms) as b:
            b.set_shape(variant, rb)
            assert b.advance(21).steps == 21
        for sc, d, want in zip(scs, doms, solo):
            got = [d.download(f) for f in ("h", "qx", "qy", "maxh")] + [np.array(d.get_clock().simtime)]
            for f, a, w in zip(("h", "qx", "qy", "maxh", "simtime"), got, want):
                assert np.array_equal(a, w), f"{sc.name}: {f} differs in {int((a != w).sum())} values"
    finally:
        for d in doms:
            d.close()
