"""The work that users of this framework have it do, as cases that can be timed.

A case is a dict of plain values; its "kind" says what a pass does:

  job       one scenario from host buffers to host buffers: upload bed,
            roughness and state, start the maximum depth, run the simulation
            to its end, download depth, discharges and maximum depth
            (a circular dam break on a flat bed, the smallest ordinary run).
  bowl      the steps between two outputs of a planar oscillation in a
            paraboloid bowl: about half of the grid is dry and the shoreline
            moves; then the download of the four output fields.
  flood     the same for a river flood in a valley: inflow hydrographs, a
            stage series at the lower edge, friction, observations every
            pass; most cells stay dry.
  rain      the same for rain on a watershed: runoff, inflows, an open
            outflow edge, every cell wet; the volume is read, too.
  ensemble  a batch of rain-on-grid members of uneven sizes, a chunk of
            batched steps as the serving loop launches them, then the
            download of every member's fields.
  kernels   one time step through the entry points that replace the
            reference's kernels one by one, on device arrays, as a host loop
            that keeps its own arrays calls them (dt read back every step).

The downloads go to pinned buffers that the caller keeps, as a program that
writes output files does.  Sizes are those of the benchmark, the tests and the
serving range (256 to 4096 a side), square and ragged.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from triton_b200 import _abi
from triton_b200.batch import Batch
from triton_b200.domain import FIELDS, Domain

GRAVITY, SQRT_G = 9.81, 3.132091953
WALL = 1e6
HEXTRA, COURANT = 0.001, 0.5
OUT = ("h", "qx", "qy", "maxh")


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # a test-sized river reach: each step is a handful of short launches
        {"name": "flood_96x150_f64", "kind": "flood", "rows": 96, "cols": 150, "prec": "fp64", "steps": 64},
        # the dam break of the reference's own example shape, start to end
        {"name": "job_512_f64", "kind": "job", "rows": 512, "cols": 512, "prec": "fp64", "seconds": 5.0},
        # the same for a ragged grid in the FP32 form
        {"name": "job_701x389_f32", "kind": "job", "rows": 701, "cols": 389, "prec": "fp32", "seconds": 5.0},
        # the benchmark's headline grid in both forms
        {"name": "bowl_2048_f64", "kind": "bowl", "rows": 2048, "cols": 2048, "prec": "fp64", "steps": 160},
        {"name": "bowl_2048_f32", "kind": "bowl", "rows": 2048, "cols": 2048, "prec": "fp32", "steps": 160},
        # a river flood on a long ragged grid, mostly dry
        {"name": "flood_1501x2750_f64", "kind": "flood", "rows": 1501, "cols": 2750, "prec": "fp64", "steps": 128},
        # rain on a watershed, every cell wet: an ordinary size in FP64, ragged
        {"name": "rain_1531x2049_f64", "kind": "rain", "rows": 1531, "cols": 2049, "prec": "fp64", "steps": 96},
        # the largest side of the serving range in the FP32 form
        {"name": "rain_4096_f32", "kind": "rain", "rows": 4096, "cols": 4096, "prec": "fp32", "steps": 96},
        # batched ensembles of uneven members in both forms
        {"name": "ensemble_24_f32", "kind": "ensemble", "members": 24, "side_min": 128, "side_max": 1024,
         "prec": "fp32", "steps": 64},
        {"name": "ensemble_10_f64", "kind": "ensemble", "members": 10, "side_min": 100, "side_max": 700,
         "prec": "fp64", "steps": 64},
        # the one-by-one kernel entries on a ragged grid
        {"name": "kernels_1000x1403", "kind": "kernels", "rows": 1000, "cols": 1403, "steps": 2},
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["job", "bowl", "flood", "rain", "ensemble", "kernels"])
    prec = rng.choice(["fp64", "fp32"])
    if kind == "ensemble":
        lo = _log(rng, 64, 256)
        return {"kind": kind, "members": _log(rng, 3, 24), "side_min": lo, "side_max": _log(rng, lo + 1, 1024),
                "prec": prec, "steps": 8 * rng.randint(2, 8)}
    if kind == "kernels":
        return {"kind": kind, "rows": _log(rng, 40, 1600), "cols": _log(rng, 40, 1600), "steps": rng.randint(1, 4)}
    rows = _log(rng, 64, 2048)
    cols = max(48, min(4096, int(rows * math.exp(rng.uniform(-0.7, 0.7)))))
    if kind == "job":
        rows, cols = min(rows, 800), min(cols, 800)
        return {"kind": kind, "rows": rows, "cols": cols, "prec": prec, "seconds": round(rng.uniform(2.0, 6.0), 2)}
    return {"kind": kind, "rows": rows, "cols": cols, "prec": prec, "steps": rng.randint(24, 128)}


# ---------------------------------------------------------------------------
# inputs, made on the GPU from the seed: padded float64 fields (ghost ring
# included, row 0 = north), forcing tables as the domain entry points take them
# ---------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _pad(a, ghost=0.0):
    return torch.nn.functional.pad(a, (1, 1, 1, 1), value=ghost)


def _edge_pad(a):
    return torch.nn.functional.pad(a[None, None], (1, 1, 1, 1), mode="replicate")[0, 0]


def _noise(g, rows, cols, octaves=8, hurst=0.8):
    out = torch.zeros((rows, cols), dtype=torch.float64, device="cuda")
    for k in range(octaves):
        n = 2 ** (k + 1) + 1
        lattice = torch.randn((1, 1, n, n), generator=g, device="cuda", dtype=torch.float64)
        out += torch.nn.functional.interpolate(lattice, size=(rows, cols), mode="bilinear",
                                               align_corners=True)[0, 0] * 2.0 ** (-hurst * k)
    return (out - out.min()) / (out.max() - out.min())


def _uniform(g, a, b):
    return a + (b - a) * float(torch.rand((), generator=g, device="cuda", dtype=torch.float64))


def _centres(rows, cols, dx):
    y = (rows - torch.arange(rows, device="cuda", dtype=torch.float64) - 0.5) * dx
    x = (torch.arange(cols, device="cuda", dtype=torch.float64) + 0.5) * dx
    return x[None, :], y[:, None]


def _inputs_job(case, g):
    R, W = case["rows"], case["cols"]
    X, Y = _centres(R, W, 1.0)
    radius = 0.1 * min(R, W) * _uniform(g, 0.9, 1.1)
    xc, yc = W * _uniform(g, 0.45, 0.55), R * _uniform(g, 0.45, 0.55)
    h = ((X - xc) ** 2 + (Y - yc) ** 2 <= radius ** 2).to(torch.float64) * _uniform(g, 8.0, 12.0)
    zero = torch.zeros_like(h)
    return dict(dx=1.0, z=_pad(zero, WALL), h=_pad(h), qx=_pad(zero), qy=_pad(zero), n2=_pad(zero))


def _inputs_bowl(case, g):
    R, W = case["rows"], case["cols"]
    n = min(R, W)
    dx = 4.0 * 2048.0 / n
    h0, a = 10.0, 3000.0
    eta, phase = a / (2 * h0) * _uniform(g, 0.4, 0.6), _uniform(g, 0.0, 2 * math.pi)
    X, Y = _centres(R, W, dx)
    xp, yp = X - 0.5 * W * dx, Y - 0.5 * R * dx
    om = math.sqrt(2 * GRAVITY * h0) / a
    z = h0 * (xp ** 2 + yp ** 2) / a ** 2
    w = h0 + (eta * h0 / a ** 2) * (2 * xp * math.cos(phase) + 2 * yp * math.sin(phase) - eta)
    h = (w - z).clamp(min=0.0)
    u, v = -eta * om * math.sin(phase), eta * om * math.cos(phase)
    return dict(dx=dx, z=_pad(z, WALL), h=_pad(h), qx=_pad(h * u), qy=_pad(h * v), n2=_pad(torch.zeros_like(h)))


def _inputs_flood(case, g):
    """A valley that falls to the east, its channel filled, the banks dry."""
    R, W = case["rows"], case["cols"]
    dx = 10.0
    r = torch.arange(R, device="cuda", dtype=torch.float64)[:, None]
    c = torch.arange(W, device="cuda", dtype=torch.float64)[None, :]
    centre = 0.5 * R + 0.12 * R * torch.sin(2 * math.pi * c / (0.5 * W) + _uniform(g, 0.0, 6.0))
    dist = (r - centre).abs() / max(R / 14.0, 4.0)
    ground = 12.0 * (1 - torch.exp(-dist ** 2)) + 2.0 * (1 - c / (W - 1)) + 3.0 * _noise(g, R, W)
    level = 3.0 + 2.0 * (1 - c / (W - 1)) + _uniform(g, 0.3, 0.6)
    h = (level - ground).clamp(min=0.0)
    qx = torch.where(h > 0.05, 0.5 * h, 0.0)
    n2 = _edge_pad(torch.exp(math.log(0.035) + 0.3 * torch.randn((R, W), generator=g, device="cuda",
                                                                dtype=torch.float64))) ** 2
    z, h, qx = _pad(ground, WALL), _pad(h), _pad(qx)
    z[1:-1, -1], h[1:-1, -1], qx[1:-1, -1] = z[1:-1, -2], h[1:-1, -2], qx[1:-1, -2]
    P = W + 2
    at = [(int(centre[0, k]), k) for k in (max(1, W // 50), max(2, W // 4))]
    peak = _uniform(g, 150.0, 250.0)
    edge = np.array([(i + 1) * P + W for i in range(R)], np.int32)
    out = dict(dx=dx, z=z, h=h, qx=qx, qy=torch.zeros_like(h), n2=n2)
    out["sources"] = dict(cells=np.array([(i + 1) * P + k + 1 for i, k in at], np.int32),
                          times=np.array([0.0, 3600.0, 7200.0, 3.6e6]),
                          flows=np.array([[40.0, 20.0], [peak, peak / 2], [60.0, 30.0], [40.0, 20.0]]).reshape(-1))
    out["extbc"] = dict(cells=edge, types=np.full(R, 1, np.int32), start=np.zeros(R, np.int32),
                        nrows=np.full(R, 4, np.int32), var1=np.array([0.0, 1800.0, 5400.0, 3.6e6]),
                        var2=np.array([3.3, 3.9, 3.5, 3.4]))
    out["obs"] = np.array([(int(centre[0, k]) + 1) * P + k + 1 for k in
                           (np.linspace(0.05, 0.95, 12) * (W - 1)).astype(int)], np.int32)
    return out


def _inputs_rain(case, g, dx=10.0, sources=2, rain=None):
    """A watershed under a film of rain, its valley filled, open to the south."""
    R, W = case["rows"], case["cols"]
    relief = 30.0 * dx * min(R, W) / 1000.0
    r = torch.arange(R, device="cuda", dtype=torch.float64)[:, None]
    c = torch.arange(W, device="cuda", dtype=torch.float64)[None, :]
    dem = relief * (0.7 * _noise(g, R, W) + 0.3 * (1 - r / (R - 1)))
    xc = 0.5 * W + 0.15 * W * torch.sin(2 * math.pi * r / (0.6 * R))
    carve = torch.exp(-((c - xc).abs() / max(W / 64.0, 3.0)) ** 2)
    dem = (dem - 0.13 * relief * carve).clamp(min=0.0)
    h = 0.002 + 0.004 * torch.rand((R, W), generator=g, device="cuda", dtype=torch.float64) + 0.8 * carve ** 2
    n2 = _edge_pad(torch.exp(math.log(0.035 * _uniform(g, 0.7, 1.3)) + 0.3 * torch.randn(
        (R, W), generator=g, device="cuda", dtype=torch.float64))) ** 2
    z, h = _pad(dem, WALL), _pad(h)
    z[-1, 1:-1], h[-1, 1:-1] = z[-2, 1:-1], h[-2, 1:-1]
    z[-2, 0] = z[-1, 0] = z[-2, 1]
    z[-2, -1] = z[-1, -1] = z[-2, -2]
    h[-2, 0], h[-2, -1] = h[-2, 1], h[-2, -2]
    P = W + 2
    out = dict(dx=dx, z=z, h=h, qx=torch.zeros_like(h), qy=torch.zeros_like(h), n2=n2)
    if sources:
        rows = np.linspace(0.1 * R, 0.45 * R, sources).astype(int)
        flows = np.zeros((4, sources))
        flows[0], flows[1] = 50.0, _uniform(g, 300.0, 500.0)
        out["sources"] = dict(cells=np.array([(int(i) + 1) * P + int(xc[int(i), 0]) + 1 for i in rows], np.int32),
                              times=np.array([0.0, 7200.0, 14400.0, 3.6e6]), flows=flows.reshape(-1))
    rate = rain if rain is not None else _uniform(g, 40.0, 60.0)
    out["runoff"] = dict(zone=np.zeros((R + 2, W + 2), np.int32), times=np.array([0.0, 3600.0, 21600.0]),
                         rates=np.array([rate, 0.0, 0.0]) / 3600.0 * 0.001, nzones=1)
    out["extbc"] = dict(cells=np.array([R * P + k + 1 for k in range(W)], np.int32), types=np.zeros(W, np.int32),
                        start=np.zeros(W, np.int32), nrows=np.ones(W, np.int32), var1=np.zeros(1), var2=np.zeros(1))
    return out


def _members(case, g):
    lo, hi = math.log(case["side_min"]), math.log(case["side_max"])
    n = case["members"]
    out = []
    for i in range(n):  # sides spread evenly over the logarithm, so that a case's work does not hang on its seed
        side = int(round(math.exp(lo + (hi - lo) * (i + 0.5) / n)))
        out.append(_inputs_rain({"rows": side, "cols": side}, g, dx=_uniform(g, 5.0, 20.0), sources=0,
                                rain=_uniform(g, 10.0, 100.0)))
    return out


def _inputs(case, seed):
    g = _gen(seed)
    if case["kind"] == "ensemble":
        return _members(case, g)
    if case["kind"] == "kernels":
        return _inputs_rain(case, g)
    return {"job": _inputs_job, "bowl": _inputs_bowl, "flood": _inputs_flood, "rain": _inputs_rain}[case["kind"]](
        case, g)


# ---------------------------------------------------------------------------
# what a user's program has in hand, and one pass
# ---------------------------------------------------------------------------
_DP = C.POINTER(C.c_double)


def _ptr(t):
    assert t.dtype == torch.float64 and t.is_contiguous() and not t.is_cuda
    return C.cast(t.data_ptr(), _DP)


def _put(d, name, t):
    _abi.check(_abi.lib().tri_domain_upload(d._h, FIELDS[name], _ptr(t), t.numel()))


def _get(d, name, t):
    _abi.check(_abi.lib().tri_domain_download(d._h, FIELDS[name], _ptr(t), t.numel()))


def _domain(s, prec):
    rows, cols = s["h"].shape
    d = Domain(rows, cols, s["dx"], COURANT, HEXTRA, 0, prec)
    for k in ("z", "n2", "h", "qx", "qy"):
        t = s[k].cpu()
        _put(d, k, t)
    _abi.check(_abi.lib().tri_domain_init_max_depth(d._h))
    if "runoff" in s:
        r = s["runoff"]
        d.set_runoff(r["zone"], r["times"], r["rates"], r["nzones"])
    if "sources" in s:
        d.set_sources(s["sources"]["cells"], s["sources"]["times"], s["sources"]["flows"])
    if "extbc" in s:
        e = s["extbc"]
        d.set_extbc(e["cells"], e["types"], e["start"], e["nrows"], e["var1"], e["var2"])
    if "obs" in s:
        d.set_observations(s["obs"])
    d.set_clock(simtime=0.0, sim_duration=1e300, print_interval=1e300, print_observation=1e300, last_obs_time=0.0,
                init_dt=0.01, time_step=0.01, it_print=0)
    return d


def _pinned(*shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=True)


def prepare(case, seed):
    s = _inputs(case, seed)
    kind = case["kind"]
    if kind == "ensemble":
        doms = [_domain(m, case["prec"]) for m in s]
        return {"case": case, "doms": doms, "batch": Batch(doms),
                "out": [_pinned(4, *m["h"].shape) for m in s]}
    if kind == "kernels":
        f = {k: s[k].contiguous() for k in ("h", "qx", "qy", "z", "n2")}
        n = f["h"].numel()
        f["maxh"] = f["h"].clone()
        for k in ("sqrth", "dt", "a0", "a1", "a2", "b0", "b1", "b2"):
            f[k] = torch.zeros(n, dtype=torch.float64, device="cuda")
        f["min"] = torch.zeros(1, dtype=torch.float64, device="cuda")
        dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
        so, ro, e = s["sources"], s["runoff"], s["extbc"]
        f.update(src=dev(so["cells"]), src_t=dev(so["times"]), src_v=dev(so["flows"]), zone=dev(ro["zone"]),
                 rate=dev(ro["rates"]), bc=dev(e["cells"]), bc_type=dev(e["types"]), bc_start=dev(e["start"]),
                 bc_rows=dev(e["nrows"]), bc_v1=dev(e["var1"]), bc_v2=dev(e["var2"]))
        return {"case": case, "dx": s["dx"], "time": 0.0, "f": f, "nsrc": so["cells"].size, "nbc": e["cells"].size}
    d = _domain(s, case["prec"])
    out = _pinned(4, *s["h"].shape)
    st = {"case": case, "dom": d, "out": out}
    if kind == "job":
        st["in"] = {k: _pinned(*s[k].shape).copy_(s[k]) for k in ("z", "n2", "h", "qx", "qy")}
    return st


def run(state):
    kind = state["case"]["kind"]
    if kind == "ensemble":
        return _run_ensemble(state)
    if kind == "kernels":
        return _run_kernels(state)
    d, out = state["dom"], state["out"]
    if kind == "job":
        for k in ("z", "n2", "h", "qx", "qy"):
            _put(d, k, state["in"][k])
        _abi.check(_abi.lib().tri_domain_init_max_depth(d._h))
        end = state["case"]["seconds"]
        d.set_clock(simtime=0.0, sim_duration=end, print_interval=end, print_id=0, it_count=0, average_dt=0.0)
        d.advance(1 << 30)
    else:
        d.advance(state["case"]["steps"])
    r = {}
    if kind == "flood":
        r["obs"] = list(d.observe())
    if kind == "rain":
        r["volume"] = np.array([d.volume()])
    for i, k in enumerate(OUT):
        _get(d, k, out[i])
    r["fields"] = [out[i] for i in range(4)]
    return r


def _run_ensemble(state):
    b = state["batch"]
    left = state["case"]["steps"]
    while left > 0:  # the serving loop's chunks
        n = min(32, left)
        b.launch(n)
        b.wait()
        left -= n
    for d, out in zip(state["doms"], state["out"]):
        for i, k in enumerate(OUT):
            _get(d, k, out[i])
    return state["out"]


def _run_kernels(state):
    """The loop body of a host that keeps its own device arrays and calls
    every kernel of a step, on torch's current stream."""
    L, f, dx = _abi.lib(), state["f"], state["dx"]
    R, W = f["h"].shape
    n = R * W
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    p = {k: C.c_void_p(v.data_ptr()) for k, v in f.items()}
    rhs = [p[k] for k in ("a0", "b0", "a1", "b1", "a2", "b2")]
    ok = _abi.check
    for _ in range(state["case"]["steps"]):
        ok(L.tri_kernel_compute_dt_and_sqrt_f64(n, dx, p["qx"], p["qy"], p["h"], p["sqrth"], p["dt"], COURANT, HEXTRA,
                                                stream))
        ok(L.tri_kernel_find_min_dt_f64(n, p["dt"], p["min"], stream))
        dt = f["min"].item()
        t = state["time"]
        ok(L.tri_kernel_flux_x_f64(n, R, W, dx, dt, p["h"], p["qx"], p["qy"], p["z"], p["sqrth"], *rhs, HEXTRA,
                                   stream))
        ok(L.tri_kernel_flux_y_f64(n, R, W, dx, dt, p["h"], p["qx"], p["qy"], p["z"], p["sqrth"], *rhs, HEXTRA,
                                   stream))
        ok(L.tri_kernel_update_cells_f64(n, R, W, dt, p["h"], p["qx"], p["qy"], p["z"], p["n2"], *rhs, HEXTRA,
                                         stream))
        row = 0 if t <= 3600.0 else 1 if t <= 21600.0 else 2
        ok(L.tri_kernel_update_runoff_f64(n, R, W, dt, p["zone"], row, 3, p["rate"], p["h"], p["qx"], p["qy"],
                                          HEXTRA, stream))
        lo = 0 if t < 7200.0 else 1 if t < 14400.0 else 2
        ok(L.tri_kernel_compute_flow_f64(state["nsrc"], p["src_t"], p["src_v"], dx, dt, t, lo, lo + 1, p["h"],
                                         p["src"], stream))
        ok(L.tri_kernel_compute_extbc_values_f64(state["nbc"], R, W, dt, p["h"], p["qx"], p["qy"], p["z"], p["n2"],
                                                 p["bc"], p["bc_type"], p["bc_start"], p["bc_rows"], p["bc_v1"],
                                                 p["bc_v2"], t, 0, 1, stream))
        ok(L.tri_kernel_wet_dry_f64(n, R, W, dt, p["h"], p["qx"], p["qy"], p["z"], p["maxh"], HEXTRA, 1, stream))
        state["time"] = t + dt
    return [f[k] for k in OUT]


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
# Operations of one cell and step: two augmented-Roe faces of about 110 each
# (square roots and quotients counted as one), the conserved update with
# friction about 40, masks and wave speed about 15.
FLOPS_CELL = 275


def _wet_share(case):
    """Share of the cells that hold water during a pass (the others hold and
    get none, and need no work)."""
    if case["kind"] == "bowl":
        n = min(case["rows"], case["cols"])
        return min(1.0, math.pi * 3000.0 ** 2 / ((8192.0 / n) ** 2 * case["rows"] * case["cols"]))
    if case["kind"] == "job":  # the disc spreads at about 2 sqrt(g h) on the dry bed; its mean area over the run
        n = min(case["rows"], case["cols"])
        r0, v, t = 0.1 * n, 18.0, case["seconds"]
        mean = r0 * r0 + r0 * v * t + (v * t) ** 2 / 3
        return min(1.0, math.pi * mean / (case["rows"] * case["cols"]))
    return 0.3 if case["kind"] == "flood" else 1.0


def work(case):
    kind = case["kind"]
    el = 8 if case.get("prec", "fp64") == "fp64" else 4
    if kind == "ensemble":
        lo, hi, n = math.log(case["side_min"]), math.log(case["side_max"]), case["members"]
        cells = sum(math.exp(lo + (hi - lo) * (i + 0.5) / n) ** 2 for i in range(n))
    else:
        cells = case["rows"] * case["cols"]
    if kind == "job":  # dt = 0.5 dx / (sqrt(g h) + |u|): about 32 steps a second at 10 m
        steps = 32.0 * case["seconds"]
    else:
        steps = case["steps"]
    # a step: h, qx, qy read and written, bed and roughness read, maximum depth read and written
    step = 10 * el * cells * _wet_share(case)
    copies = 0 if kind == "kernels" else 4 * 8 * cells
    if kind == "job":
        copies += 5 * 8 * cells
    return {"bytes": step * steps + copies, "flops": FLOPS_CELL * cells * _wet_share(case) * steps}


# ---------------------------------------------------------------------------
# the same passes in plain torch, 64 bits
# ---------------------------------------------------------------------------
def _velocity(h, q):
    return torch.where(h >= HEXTRA, q / torch.where(h >= HEXTRA, h, 1.0), 0.0)


def _face(a, b, x, dx, dt):
    """Contributions of the faces between cells a (owners) and b, each a tuple
    (h, qx, qy, z); x: faces with normal (1, 0), else (0, 1).  Augmented Roe
    solver with an entropy fix, a limited bed-step source and the redirection
    of mass from dry sides."""
    h1, qx1, qy1, z1 = a
    h2, qx2, qy2, z2 = b
    wet = (h1 > 0) | (h2 > 0)
    one, nil = torch.ones_like(h1), torch.zeros_like(h1)
    s1, s2 = h1.sqrt(), h2.sqrt()
    u1, v1, u2, v2 = _velocity(h1, qx1), _velocity(h1, qy1), _velocity(h2, qx2), _velocity(h2, qy2)
    h12, dh = torch.where(wet, 0.5 * (h1 + h2), one), h2 - h1
    c = (GRAVITY * h12).sqrt()
    ss = torch.where(wet, s1 + s2, one)
    u, v = (u1 * s1 + u2 * s2) / ss, (v1 * s1 + v2 * s2) / ss
    un, un1, un2 = (u, u1, u2) if x else (v, v1, v2)
    l0, l1, l2 = un - c, un, un + c
    e1, e2 = un1 - SQRT_G * s1, un2 - SQRT_G * s2
    fix = (e1 < 0) & (e2 > 0)
    t = e1 * (e2 - l0) / torch.where(fix, e2 - e1, one)
    le0, l0 = torch.where(fix, l0 - t, nil), torch.where(fix, t, l0)
    e1, e2 = un1 + SQRT_G * s1, un2 + SQRT_G * s2
    fix = (e1 < 0) & (e2 > 0)
    t = e2 * (l2 - e1) / torch.where(fix, e2 - e1, one)
    le2, l2 = torch.where(fix, l2 - t, nil), torch.where(fix, t, l2)
    r01, r02 = (u - c, v) if x else (u, v - c)
    r21, r22 = (u + c, v) if x else (u, v + c)
    dqx, dqy = qx2 - qx1, qy2 - qy1
    aq = ((dqx if x else dqy) - un * dh) / c
    al0, al2 = 0.5 * (dh - aq), 0.5 * (dh + aq)
    al1 = ((dqy - v * dh) if x else -(dqx - u * dh)) / c
    dz = z2 - z1
    dzp = torch.where(dz >= 0, torch.where(z1 + h1 < z2, h1, dz), torch.where(z2 + h2 < z1, -h2, dz))
    hp = torch.where(dz >= 0, h1, h2)
    be = 0.5 * GRAVITY * (hp - 0.5 * dzp.abs()) * dzp / c
    hp = h1 + al0
    lim = (l0 * l2 < 0) & (hp > 0) & (h1 > 0) & (h2 > 0)
    f0 = torch.where(lim, l0, one) / torch.where(lim, l0 + le2, one)
    f2 = torch.where(lim, l2, one) / torch.where(lim, l2 + le0, one)
    low = torch.maximum(be, f0 * (al0 * l0 - h1 * dx * 0.5 / dt + le2 * h2))
    low = torch.minimum(low, f2 * (-al2 * l2 + h2 * dx * 0.5 / dt + le0 * h1))
    be = torch.where(lim, low, be)
    w0, w1, w2 = l0 * al0 - be, l1 * al1, l2 * al2 + be
    p, q = [nil, nil, nil], [nil, nil, nil]

    def add(w, sign, vec):
        for k, r in enumerate(vec):
            if r is None:
                continue
            q[k] = q[k] + torch.where(sign, w * r, nil)
            p[k] = p[k] + torch.where(sign, nil, w * r)

    add(w0, l0 > 0, (one, r01, r02))
    add(w1, l1 > 0, (None, None, c) if x else (None, -c, None))
    add(w2, l2 > 0, (one, r21, r22))
    dry2 = (h2 < 1e-12) & (hp - be / torch.where(l2 != 0, l2, one) < -1e-12)
    dry1 = ~dry2 & (h1 < 1e-12) & (hp - be / torch.where(l0 != 0, l0, one) < -1e-12)
    both = w0 + w2
    p = [torch.where(dry2, both if k == 0 else nil, torch.where(dry1, nil, p[k])) for k in range(3)]
    q = [torch.where(dry1, both if k == 0 else nil, torch.where(dry2, nil, q[k])) for k in range(3)]
    add(le0 * al0, le0 > 0, (one, r01, r02))
    add(le2 * al2, le2 > 0, (one, r21, r22))

    def scaled(v):
        return torch.where(wet & (v.abs() >= 1e-12), dt * v / dx, nil)

    return [scaled(v) for v in p], [scaled(v) for v in q]


def _largest_speed(s):
    h, m = s["h"], s["h"] > HEXTRA
    d = torch.maximum(s["qx"].abs(), s["qy"].abs()) / torch.where(m, h, 1.0) + SQRT_G * h.sqrt()
    return float(torch.where(m, d, 0.0).max())


def _bracket(times, t):
    n = len(times)
    for i in range(n - 1):
        if times[i + 1] > t:
            return i, i + 1
    return n - 1, n - 1


def _step(s, t, dt):
    h, qx, qy, z, n2 = (s[k] for k in ("h", "qx", "qy", "z", "n2"))
    dx = s["dx"]
    part = lambda r, c: tuple(a[r, c] for a in (h, qx, qy, z))  # noqa: E731
    mid = slice(1, -1)
    xa, xb = _face(part(mid, slice(None, -1)), part(mid, slice(1, None)), True, dx, dt)
    ya, yb = _face(part(slice(1, None), mid), part(slice(None, -1), mid), False, dx, dt)
    inner = lambda a: a[1:-1, 1:-1]  # noqa: E731
    hn = inner(h)
    new = [(inner(a) - (xa[k][:, 1:] + ya[k][:-1])) - (xb[k][:, :-1] + yb[k][1:]) for k, a in enumerate((h, qx, qy))]
    del xa, xb, ya, yb
    hij = new[0].clamp(min=0.0)
    mx, my = new[1], new[2]
    mod = (mx * mx + my * my).sqrt()
    rough = (inner(n2) > 1e-12) & (hn >= HEXTRA) & (mod > 1e-12)
    hs = torch.where(rough, hn, 1.0)
    tt = torch.where(rough, dt * GRAVITY * inner(n2) * mod / (hs * hs * hs.pow(1.0 / 3.0)), 1.0)
    k = torch.where(rough, 2.0 / (1.0 + (1.0 + 4.0 * tt).sqrt()), 1.0)  # the root, without its cancellation
    ok = hij >= HEXTRA
    mx, my = torch.where(ok, mx * k, 0.0), torch.where(ok, my * k, 0.0)
    if "runoff" in s:
        ro = s["runoff"]
        rate = float(ro["rates"][min(_row(ro["times"], t), len(ro["rates"]) - 1)])
        hij = hij + rate * dt
        low = hij < HEXTRA
        hij = hij.clamp(min=0.0)
        mx, my = torch.where(low, 0.0, mx), torch.where(low, 0.0, my)
    h[1:-1, 1:-1], qx[1:-1, 1:-1], qy[1:-1, 1:-1] = hij, mx, my
    if "sources" in s:
        so = s["sources"]
        lo, hi = _bracket(so["times"], t)
        v = so["flows"].reshape(len(so["times"]), -1)
        w = 0.0 if lo == hi else (t - so["times"][lo]) / (so["times"][hi] - so["times"][lo])
        for i, cell in enumerate(so["cells"]):
            h.view(-1)[int(cell)] += (v[lo, i] + (v[hi, i] - v[lo, i]) * w) * dt / (dx * dx)
    if "extbc" in s and s["extbc"]["types"][0] == 0:  # open southern edge
        for a in (h, qx, qy):
            a[-1, 1:-1] = a[-2, 1:-1]
            a[-2, 0], a[-2, -1] = a[-2, 1].clone(), a[-2, -2].clone()
    elif "extbc" in s:  # stage series along the eastern edge; its corner cells are at rest
        e = s["extbc"]
        tm = 0.5 * (t + t + dt)
        level = float(np.interp(tm, e["var1"], e["var2"]))
        h[1:-1, -2] = (level - z[1:-1, -2]).clamp(min=0.0)
        qy[1:-1, -2] = 0.0
        qx[1, -2] = qx[-2, -2] = 0.0
        for a in (h, qx, qy):
            a[1:-1, -1] = a[1:-1, -2]
            a[0, -2], a[-1, -2] = a[1, -2].clone(), a[-2, -2].clone()
    hc, zc, m = inner(h), inner(z), inner(h) > HEXTRA
    lvl = hc + zc
    stop = lambda hb, zb: (lvl < zb) & (hb < 1e-12)  # noqa: E731
    sx = m & (stop(h[1:-1, 2:], z[1:-1, 2:]) | stop(h[1:-1, :-2], z[1:-1, :-2]))
    sy = m & (stop(h[:-2, 1:-1], z[:-2, 1:-1]) | stop(h[2:, 1:-1], z[2:, 1:-1]))
    inner(qx).masked_fill_(sx, 0.0)
    inner(qy).masked_fill_(sy, 0.0)
    inner(s["maxh"]).copy_(torch.maximum(inner(s["maxh"]), hc))


def _row(times, t):
    return int(np.searchsorted(np.asarray(times), t, side="left")) - 1 if t > times[0] else 0


def _advance(s, steps=None, end=None):
    s["maxh"] = s["h"].clone()
    t, k = 0.0, 0
    while (steps is not None and k < steps) or (end is not None and t < end):
        top = _largest_speed(s)
        dt = COURANT * s["dx"] / top if top > 0 else 0.01
        if end is not None and t + dt > end:
            dt = end - t
        _step(s, t, dt)
        t += dt
        k += 1


def exact(case, seed):
    """What run() returns for these inputs after its first pass."""
    s = _inputs(case, seed)
    kind = case["kind"]
    if kind == "ensemble":
        out = []
        for m in s:
            _advance(m, steps=case["steps"])
            out.append(torch.stack([m[k] for k in OUT]).cpu())
        return out
    _advance(s, steps=case.get("steps"), end=case.get("seconds"))
    if kind == "kernels":
        return [s[k] for k in OUT]
    r = {"fields": [s[k].cpu() for k in OUT]}
    if kind == "flood":
        at = torch.from_numpy(s["obs"].astype(np.int64)).cuda()
        r["obs"] = [s[k].view(-1)[at].cpu().numpy() for k in ("h", "qx", "qy")]
    if kind == "rain":
        r["volume"] = np.array([float(s["h"][1:-1, 1:-1].sum()) * s["dx"] ** 2])
    return r
