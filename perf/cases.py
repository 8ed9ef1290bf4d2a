"""The work whose speed counts, as cases that a measurement can run.

A case is a dict of plain values; ``kind`` names the entry point it goes through:

* ``screen``: ``mzb_conjunctions`` on a polyjectory that is already in HBM, the
  results copied into the program's device buffers with the
  ``mzb_result_copy_*`` accessors, as a program does that goes on working with
  them on the GPU.  ``form`` is the screening form ("plain" is the default of
  the entry points);
* ``files``: the drop-in class ``conjunctions``, which leaves its results in the
  memory-mapped files of a private directory;
* ``states``: ``polyjectory.state_eval`` (``times`` 0: one time for all objects)
  or ``polyjectory.state_meval`` into the caller's host array;
* ``propagate``: ``mzb_sgp4_propagate`` between device arrays;
* ``produce``: ``mzb_make_sgp4_polyjectory``, element sets to a polyjectory whose
  coefficients go to device memory (to be screened there) and whose times and
  offsets go to host memory.

Buffers for results of varying length have a size that the case alone gives;
the counts come with them.

The catalogues are the seeded ones of ``mizuba_b200.synth``: 80 % LEO, 15 %
MEO / HEO and 5 % GEO, optionally with circular dense shells (``shells``
objects) or a share of low, fast-decaying orbits (``lowp``).
"""

import ctypes as ct
import math

import numpy as np
import torch

import mizuba_b200 as mz
from mizuba_b200 import _native, synth

MINUTE = 1.0 / 1440.0
JD0 = 2460496.5  # 0h UTC, 5 July 2024


def _screen(name, n, days, thresh, form, shells=0, lowp=0.0, order=18, interval=3.0, masked=False):
    return {"name": name, "kind": "screen", "objects": n, "days": days, "thresh": thresh, "form": form,
            "shells": shells, "lowp": lowp, "order": order, "interval": interval, "masked": masked}


def listed():
    return [
        # The smallest call: an operator screens a handful of objects over a
        # few hours with a wide threshold.  Launches and read-backs count.
        _screen("screen_150_3h_plain", 150, 0.125, 80.0, "plain"),
        # A constellation's own day (the 1,000-object day of the benchmark).
        _screen("screen_1k_day_plain", 1000, 1.0, 5.0, "plain"),
        # The catalogue day, all FP64: the default form on the headline size.
        _screen("screen_20k_day_plain", 20000, 1.0, 5.0, "plain"),
        # The same in the faster form: the benchmark's headline.
        _screen("screen_20k_day_mixed", 20000, 1.0, 5.0, "mixed"),
        # Dense shells at 10 km: many candidate pairs per object.
        _screen("screen_20k_shells_mixed", 20000, 0.4, 10.0, "mixed", shells=6000),
        # The stress catalogue at 20 km: pairs, items and records dominate.
        _screen("screen_60k_shells_20km_mixed", 60000, 0.1, 20.0, "mixed", shells=15000),
        # A week's catalogue has many low, drag-shortened segments; a first
        # slice of it, in the default form, objects of all three types.
        _screen("screen_30k_lowp_types_plain", 29989, 0.2, 5.0, "plain", lowp=0.05, masked=True),
        # Higher order, odd sizes and an interval that does not divide the span.
        _screen("screen_order25_odd_plain", 3001, 0.3, 20.0, "plain", order=25, interval=2.3),
        # The drop-in class with its output files, at a working size.
        {"name": "files_2k_6h_plain", "kind": "files", "objects": 2000, "days": 0.25, "thresh": 10.0,
         "form": "plain", "shells": 0, "lowp": 0.0, "order": 18, "interval": 3.0, "masked": False},
        # Ephemerides: every minute of half a day for a few thousand objects.
        {"name": "states_3k_720", "kind": "states", "objects": 3000, "days": 0.5, "times": 720, "shells": 0,
         "lowp": 0.0, "order": 18},
        # Look angles and pass predictions: a catalogue at many instants.
        {"name": "propagate_8k_144", "kind": "propagate", "sets": 8000, "times": 144, "span_min": 1440.0},
        # A catalogue's element sets turned into trajectories.
        {"name": "produce_6k_6h", "kind": "produce", "sets": 6000, "days": 0.25, "per_object": 1},
    ]


def _log(rng, a, b):
    return math.exp(rng.uniform(math.log(a), math.log(b)))


def draw(rng):
    kind = rng.choice(["screen"] * 6 + ["files", "states", "propagate", "produce"])
    if kind in ("screen", "files"):
        n = int(_log(rng, 100, 24000 if kind == "screen" else 2500))
        days = min(1.0, _log(rng, 0.05, 1.0), (5000.0 if kind == "screen" else 400.0) / n)
        shells = int(n * rng.uniform(0.1, 0.4)) if rng.random() < 0.35 else 0
        thresh = round(_log(rng, 2.0, 20.0 if n > 4000 else 60.0), 2)
        return {"kind": kind, "objects": n, "days": round(days, 3), "thresh": thresh,
                "form": rng.choice(["plain", "mixed"]), "shells": shells,
                "lowp": rng.choice([0.0, 0.0, 0.05]), "order": rng.choice([18] * 6 + [12, 15, 20, 25]),
                "interval": rng.choice([3.0, 3.0, round(rng.uniform(1.0, 9.0), 2)]), "masked": rng.random() < 0.3}
    if kind == "states":
        n = int(_log(rng, 50, 6000))
        times = 0 if rng.random() < 0.25 else int(min(_log(rng, 2, 1500), 2.2e6 / n))
        return {"kind": kind, "objects": n, "days": round(rng.uniform(0.1, 0.5), 3), "times": times, "shells": 0,
                "lowp": 0.0, "order": rng.choice([18, 18, 18, 12, 25])}
    if kind == "propagate":
        n = int(_log(rng, 20, 10000))
        return {"kind": kind, "sets": n, "times": int(max(1, min(_log(rng, 4, 2000), 1.2e6 / n))),
                "span_min": round(_log(rng, 60.0, 2880.0), 1)}
    n = int(_log(rng, 30, 6000))
    return {"kind": "produce", "sets": n, "days": round(min(_log(rng, 0.1, 1.0), 1500.0 / n), 3),
            "per_object": rng.choice([1, 1, 3])}


# ------------------------------------------------------------------ inputs


def _elements(case, rng):
    el = synth.base_elements(case["objects"] - case["shells"], rng, case["lowp"])
    if case["shells"]:
        el = np.concatenate([el, synth.shell_elements(case["shells"], rng)])
    return el


def _polyjectory(case, seed):
    rng = np.random.default_rng(seed)
    pj = synth.build_polyjectory(_elements(case, rng), case["days"], order=case["order"])
    types = None
    if case.get("masked"):
        types = rng.choice(np.array([1, 2, 4], dtype=np.int32), pj.n_objs, p=[0.7, 0.2, 0.1])
        types[0] = 1  # at least one primary: the screen is not skipped
    return pj, types, rng


def _gpes(n, per_object, rng):
    """Element sets of n / per_object objects, epochs in the day before JD0
    and, for several sets an object, in the hours after it."""
    objs = max(1, n // per_object)
    el = synth.base_elements(objs, rng, 0.0)
    g = np.zeros(objs * per_object, dtype=mz.gpe_dtype)
    for k in range(per_object):
        rows = g[k::per_object]
        rows["norad_id"] = np.arange(1, objs + 1)
        rows["epoch_jd1"] = JD0
        rows["epoch_jd2"] = rng.uniform(-1.0, 0.0, objs) if k == 0 else 0.03 * k + rng.uniform(0.0, 0.02, objs)
        rows["n0"] = 60.0 * np.sqrt(398600.8 / el[:, 0] ** 3)  # rad / min, WGS72
        rows["e0"], rows["i0"], rows["node0"], rows["omega0"] = el[:, 1], el[:, 2], el[:, 3], el[:, 4]
        rows["m0"] = np.mod(el[:, 5] + rows["n0"] * 1440.0 * rows["epoch_jd2"], 2 * np.pi)
        rows["bstar"] = el[:, 6]
    return g


def _steps(case):
    return math.ceil(case["days"] / (case["interval"] * MINUTE) - 1e-9)


def _pairs(case):
    """About as many broad-phase pairs as the case has."""
    n = case["objects"]
    dense = 1 + 60 * (case["shells"] / n) ** 2 * max(1.0, case["thresh"] / 10)
    return 2.4e-5 * n * n * _steps(case) * dense * (case["interval"] / 3) ** 2 * (1 + case["thresh"] / 100)


def _room(case):
    """Buffer sizes: tree nodes, pairs and conjunction records."""
    pairs = int(6 * _pairs(case)) + 4 * case["shells"] * _steps(case) + 8192
    return _steps(case) * (2 * case["objects"] - 1), pairs, pairs // 16 + 1024


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("screen", "files"):
        pj, types, _ = _polyjectory(case, seed)
        dev = mz.to_device(pj)
        n, s = case["objects"], _steps(case)
        nodes, pairs, conjs = _room(case)
        if kind == "files":
            return {"case": case, "pj": pj, "types": types, "trees": np.zeros(nodes, mz.conjunctions.bvh_node),
                    "pairs": np.zeros(pairs, mz.conjunctions.aabb_collision),
                    "conj": np.zeros(conjs, mz.conjunctions.conj)}
        opts = _native.MzbOpts()
        opts.form = 1 if case["form"] == "mixed" else 0
        z = lambda *shape, dtype=torch.int32: torch.zeros(shape, dtype=dtype, device="cuda")  # noqa: E731
        # The screen needs the polyjectory in HBM only.
        return {"case": case, "dev": dev, "types": types, "opts": opts, "room": (nodes, pairs, conjs),
                "aabbs": z(s, n + 1, 2, 4, dtype=torch.float32), "srt_aabbs": z(s, n + 1, 2, 4, dtype=torch.float32),
                "mcodes": z(s, n, dtype=torch.int64), "srt_mcodes": z(s, n, dtype=torch.int64), "srt_idx": z(s, n),
                "trees": z(nodes, 12), "pairs": z(pairs, 2), "conj": z(conjs, 30),
                "tree_offsets": np.zeros((s, 2), np.uint64), "bp_offsets": np.zeros((s, 2), np.uint64)}
    if kind == "states":
        pj, _, rng = _polyjectory(case, seed)
        mz.to_device(pj)
        n, t = case["objects"], case["times"]
        # Some requests lie outside the data, as a user's do at the span's ends.
        tm = float(rng.uniform(0.0, case["days"])) if t == 0 else np.sort(rng.uniform(-0.001, case["days"] * 1.002, t))
        return {"case": case, "pj": pj, "time": tm, "out": np.zeros((n, 7) if t == 0 else (n, t, 7))}
    rng = np.random.default_rng(seed)
    if kind == "propagate":
        g = _gpes(case["sets"], 1, rng)
        n, t = len(g), case["times"]
        return {"case": case, "n": n, "t": t,
                "gpes": torch.from_numpy(g.view(np.uint8).copy()).cuda(),
                "tsince": torch.from_numpy(np.sort(rng.uniform(0.0, case["span_min"], t))).cuda(),
                "out": torch.zeros((n, t, 6), dtype=torch.float64, device="cuda"),
                "err": torch.zeros((n, t), dtype=torch.int32, device="cuda")}
    g = _gpes(case["sets"], case["per_object"], rng)
    objs = len(g) // case["per_object"]
    room = int(objs * (case["days"] * 260 + 8 * case["per_object"])) + 4096  # segments
    return {"case": case, "gpes": g, "room": room, "traj": torch.zeros(room * 133, dtype=torch.float64, device="cuda"),
            "traj_offsets": np.zeros((objs, 2), np.uint64), "time": np.zeros(room + objs),
            "time_offsets": np.zeros(objs, np.uint64), "status": np.zeros(objs, np.int32)}


# ------------------------------------------------------------------ passes


def _ok(L, rc):
    if rc != 0:
        raise RuntimeError(L.mzb_last_error().decode())


def _run_screen(st):
    c, L = st["case"], _native.core()
    res = ct.c_void_p()
    types = st["types"]
    _ok(L, L.mzb_conjunctions(st["dev"]._h, c["thresh"], c["interval"] * MINUTE,
                              None if types is None else types.ctypes.data, ct.byref(st["opts"]), ct.byref(res)))
    try:
        nodes, pairs, conjs = (int(getattr(L, "mzb_result_n_" + w)(res)) for w in ("tree_nodes", "bp", "conj"))
        if nodes > st["room"][0] or pairs > st["room"][1] or conjs > st["room"][2]:
            raise RuntimeError("the result buffers are too small")
        for name in ("aabbs", "srt_aabbs", "mcodes", "srt_mcodes", "srt_idx", "trees", "conj"):
            _ok(L, getattr(L, "mzb_result_copy_" + name)(res, st[name].data_ptr()))
        _ok(L, L.mzb_result_copy_bp(res, st["pairs"].data_ptr()))
        _ok(L, L.mzb_result_tree_offsets(res, st["tree_offsets"].ctypes.data))
        _ok(L, L.mzb_result_bp_offsets(res, st["bp_offsets"].ctypes.data))
    finally:
        L.mzb_result_free(res)
    rec = st["conj"].view(torch.float64)
    out = {name: st[name] for name in ("aabbs", "srt_aabbs", "mcodes", "srt_mcodes", "srt_idx", "pairs")}
    out |= {"tree_links": st["trees"][:, :4], "tree_boxes": st["trees"].view(torch.float32)[:, 4:],
            "tree_offsets": st["tree_offsets"].view(np.int64), "bp_offsets": st["bp_offsets"].view(np.int64),
            "counts": [nodes, pairs, conjs],
            "conj": {"ij": st["conj"][:, :2], "tca": rec[:, 1], "dca": rec[:, 2], "ri": rec[:, 3:6],
                     "vi": rec[:, 6:9], "rj": rec[:, 9:12], "vj": rec[:, 12:15]}}
    return out


def _run_files(st):
    c = st["case"]
    r = mz.conjunctions(st["pj"], c["thresh"], c["interval"] * MINUTE, otypes=st["types"], form=c["form"])
    trees, pairs, conj, nodes, n_pairs = st["trees"], st["pairs"], st["conj"], 0, 0
    for k in range(r.n_cd_steps):
        t, p = r.get_bvh_tree(k), r.get_aabb_collisions(k)
        trees[nodes:nodes + len(t)] = t
        pairs[n_pairs:n_pairs + len(p)] = p
        nodes, n_pairs = nodes + len(t), n_pairs + len(p)
    rec = r.conjunctions
    conj[:len(rec)] = rec
    links = trees.view(np.int32).reshape(-1, 12)
    return {"aabbs": r.aabbs, "srt_aabbs": r.srt_aabbs, "mcodes": r.mcodes.view(np.int64),
            "srt_mcodes": r.srt_mcodes.view(np.int64), "srt_idx": r.srt_idx.view(np.int32),
            "pairs": pairs.view(np.int32), "tree_links": links[:, :4],
            "tree_boxes": links[:, 4:].view(np.float32), "counts": [nodes, n_pairs, len(rec)],
            "conj": {"ij": conj.view(np.int32).reshape(-1, 30)[:, :2], **{f: conj[f] for f in (
                "tca", "dca", "ri", "vi", "rj", "vj")}}}


def _run_produce(st):
    g, L = st["gpes"], _native.core()
    h = ct.c_void_p()
    _ok(L, L.mzb_make_sgp4_polyjectory(g.ctypes.data, len(g), JD0, JD0 + st["case"]["days"], 0.0, math.inf,
                                       ct.byref(h)))
    try:
        sizes, epoch = np.zeros(4, np.uint64), np.zeros(3)
        L.mzb_sgp4_pj_sizes(h, sizes.ctypes.data)
        L.mzb_sgp4_pj_epoch(h, epoch.ctypes.data)
        if int(sizes[1]) > st["traj"].numel() or int(sizes[2]) > len(st["time"]):
            raise RuntimeError("the result buffers are too small")
        _ok(L, L.mzb_sgp4_pj_copy(h, st["traj"].data_ptr(), st["traj_offsets"].ctypes.data, st["time"].ctypes.data,
                                  st["time_offsets"].ctypes.data, st["status"].ctypes.data))
    finally:
        L.mzb_sgp4_pj_free(h)
    return {"traj": st["traj"], "traj_offsets": st["traj_offsets"].view(np.int64), "time": st["time"],
            "time_offsets": st["time_offsets"].view(np.int64), "status": st["status"],
            "sizes": sizes.view(np.int64), "epoch": epoch}


def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "screen":
        return _run_screen(state)
    if kind == "files":
        return _run_files(state)
    if kind == "states":
        pj = state["pj"]
        f = pj.state_eval if c["times"] == 0 else pj.state_meval
        return f(state["time"], out=state["out"])
    if kind == "propagate":
        L = _native.core()
        _ok(L, L.mzb_sgp4_propagate(state["gpes"].data_ptr(), state["n"], state["tsince"].data_ptr(), state["t"],
                                    state["out"].data_ptr(), state["err"].data_ptr()))
        return {"states": state["out"], "codes": state["err"]}
    return _run_produce(state)


# ------------------------------------------------------------------ work


def work(case):
    kind = case["kind"]
    if kind in ("screen", "files"):
        n, op1 = case["objects"], case["order"] + 1
        s, pairs = _steps(case), _pairs(case)
        seg = n * case["days"] * 90  # order-18 segments of this mix: 90 per object and day
        items = n * s + seg  # segments cut at the step bounds
        # Trajectories of x, y, z, r read once; boxes, codes, indices and trees
        # written once and in sorted order; pairs written.
        size = seg * (4 * op1 + 1) * 8 + n * s * (2 * 32 + 2 * 8 + 4 + 2 * 48) + pairs * 8
        # Enclosure of four coordinates per item: shift and difference table.
        # Half of the pairs' sub-intervals are cut once: squared distance on
        # op1 nodes, interpolation and enclosure.
        ops = items * 4 * 2 * op1 * op1 + 1.4 * pairs * (12 * op1 * op1 + 2 * op1 * op1)
        return {"bytes": size, "flops": ops}
    if kind == "states":
        n, t, op1 = case["objects"], max(1, case["times"]), case["order"] + 1
        seg = min(n * case["days"] * 90, n * t)
        return {"bytes": seg * 7 * op1 * 8 + n * t * 56, "flops": n * t * 7 * 2 * op1}
    if kind == "propagate":
        e = case["sets"] * case["times"]
        return {"bytes": e * 52 + case["sets"] * 80, "flops": e * 600}
    seg = case["sets"] // case["per_object"] * case["days"] * 130
    # 38 propagations a segment, the interpolation of 7 variables.
    return {"bytes": seg * 133 * 8, "flops": seg * (38 * 600 + 7 * 3 * 19 * 19)}


# ------------------------------------------------------------------ 64-bit values


def _states_at(a, op1, i, tm):
    """x, y, z, vx, vy, vz, r of object i at the times tm, and d/dt of x, y, z."""
    off, ns = int(a["traj_offsets"][i, 0]), int(a["traj_offsets"][i, 1])
    t = a["time"][int(a["time_offsets"][i]):][:ns + 1]
    cf = a["traj"][off:off + ns * op1 * 7].reshape(ns, op1, 7)
    k = np.searchsorted(t, tm, side="right") - 1
    inside = (k >= 0) & (tm < t[-1])
    k = np.clip(k, 0, ns - 1)
    h = (tm - t[k])[:, None]
    v, d = cf[k, op1 - 1].copy(), np.zeros((len(tm), 7))
    for o in range(op1 - 2, -1, -1):
        d = d * h + v
        v = v * h + cf[k, o]
    v[~inside] = np.nan
    return v, d[:, :3]


def _boxes(a, op1, n, days, interval, radius):
    """The Cargo-Shisha boxes of every object and step, rounded outward to
    float, with each step's global box behind them."""
    s = int(math.ceil(a["maxT"] / interval))
    box = np.empty((s, n + 1, 2, 4), dtype=np.float32)
    box[:, :, 0], box[:, :, 1] = np.inf, -np.inf
    m = op1 - 1
    binom = np.array([[math.comb(i, k) for k in range(op1)] for i in range(op1)], dtype=np.float64)
    cb = interval * np.arange(s)
    ce = np.append(interval * np.arange(1, s), a["maxT"])
    for i in range(n):
        off, ns = int(a["traj_offsets"][i, 0]), int(a["traj_offsets"][i, 1])
        if ns == 0:
            continue
        t = a["time"][int(a["time_offsets"][i]):][:ns + 1]
        cf = a["traj"][off:off + ns * op1 * 7].reshape(ns, op1, 7)[:, :, [0, 1, 2, 6]]
        lo = np.maximum(np.searchsorted(t, cb, side="right") - 1, 0)
        hi = np.minimum(np.searchsorted(t, ce, side="left"), ns)
        cnt = np.where((t[0] >= ce) | (t[-1] <= cb), 0, np.maximum(hi - lo, 0))
        st = np.repeat(np.arange(s), cnt)
        sg = np.concatenate([np.arange(l, l + k) for l, k in zip(lo, cnt)]).astype(np.int64)
        b = np.maximum(cb[st], t[sg]) - t[sg]
        delta = np.minimum(ce[st], t[sg + 1]) - t[sg] - b
        c = cf[sg]
        for p in range(m):  # Taylor shift
            for k in range(m - 1, p - 1, -1):
                c[:, k] += b[:, None] * c[:, k + 1]
        c *= (delta[:, None] ** np.arange(op1) / binom[m])[:, :, None]
        mn, mx = c[:, 0].copy(), c[:, 0].copy()
        for k in range(1, op1):
            c = c[:, :-1] + c[:, 1:]
            mn, mx = np.minimum(mn, c[:, 0]), np.maximum(mx, c[:, 0])
        fl = np.nextafter((mn - radius).astype(np.float32), np.float32(-np.inf))
        fu = np.nextafter((mx + radius).astype(np.float32), np.float32(np.inf))
        np.minimum.at(box[:, i, 0], st, fl)
        np.maximum.at(box[:, i, 1], st, fu)
    box[:, n, 0] = box[:, :n, 0].min(axis=1)
    box[:, n, 1] = box[:, :n, 1].max(axis=1)
    return box


def _close_approaches(a, op1, n, thresh, room):
    """Records of all minima of the mutual distances below the threshold, by
    dense sampling and bisection of d(d^2)/dt; pairs that are close and
    departing at the start, or approaching at the end, count as well."""
    T = a["maxT"]
    grid = np.linspace(0.0, T, int(T * 86400 / 10) + 2)
    grid[-1] = np.nextafter(T, 0.0)
    pv = [_states_at(a, op1, i, grid) for i in range(n)]
    pos, vel = np.stack([p[0][:, :3] for p in pv]), np.stack([p[1] for p in pv])
    rec = []

    def slope(i, j, t):
        (p, v), (q, w) = (_states_at(a, op1, o, np.array([t])) for o in (i, j))
        return float(np.sum((p[:, :3] - q[:, :3]) * (v - w)))

    for i in range(n - 1):
        dr, dv = pos[i] - pos[i + 1:], vel[i] - vel[i + 1:]
        f, d = np.sum(dr * dv, axis=2), np.sqrt(np.sum(dr * dr, axis=2))
        near = np.minimum(d[:, :-1], d[:, 1:]) < thresh + 90.0
        for j, k in zip(*np.nonzero((f[:, :-1] < 0) & (f[:, 1:] >= 0) & near)):
            lo, hi = grid[k], grid[k + 1]
            for _ in range(60):
                mid = (lo + hi) / 2
                lo, hi = (mid, hi) if slope(i, i + 1 + j, mid) < 0 else (lo, mid)
            rec.append((i, i + 1 + j, (lo + hi) / 2))
        rec += [(i, i + 1 + j, 0.0) for j in np.nonzero(f[:, 0] > 0)[0] if d[j, 0] < thresh]
        rec += [(i, i + 1 + j, grid[-1]) for j in np.nonzero(f[:, -1] < 0)[0] if d[j, -1] < thresh]
    out = []
    for i, j, t in sorted(rec, key=lambda r: (r[2], r[0], r[1])):
        p, q = (_states_at(a, op1, o, np.array([t]))[0][0] for o in (i, j))
        d = float(np.linalg.norm(p[:3] - q[:3]))
        if d < thresh:
            out.append(np.concatenate([[t, d], p[:6], q[:6]]))
    r = np.zeros((room, 14))
    r[:len(out)] = np.array(out).reshape(-1, 14)
    return {"ij": None, "tca": r[:, 0], "dca": r[:, 1], "ri": r[:, 2:5], "vi": r[:, 5:8], "rj": r[:, 8:11],
            "vj": r[:, 11:14]}


def exact(case, seed):
    kind = case["kind"]
    if kind == "states":
        pj, _, rng = _polyjectory(case, seed)
        n, t, op1 = case["objects"], case["times"], case["order"] + 1
        if n * max(1, t) > 4e6:
            return None
        tm = np.array([rng.uniform(0.0, case["days"])]) if t == 0 else np.sort(
            rng.uniform(-0.001, case["days"] * 1.002, t))
        v = np.stack([_states_at(pj.arrays, op1, i, tm)[0] for i in range(n)])
        return v[:, 0] if t == 0 else v
    if kind in ("screen", "files"):
        n, op1 = case["objects"], case["order"] + 1
        steps = case["days"] / (case["interval"] * MINUTE)
        # The mixed form's boxes enclose these, with a margin of its own.
        if case["form"] != "plain" or n * steps * op1 * op1 > 2.5e8:
            return None
        pj, types, _ = _polyjectory(case, seed)
        a = pj.arrays
        out = dict.fromkeys(("srt_aabbs", "mcodes", "srt_mcodes", "srt_idx", "tree_links", "tree_boxes", "pairs",
                             "counts", "conj"))
        if kind == "screen":
            out["tree_offsets"] = out["bp_offsets"] = None
        out["aabbs"] = _boxes(a, op1, n, case["days"], case["interval"] * MINUTE, case["thresh"] / 2)
        if types is None and n <= 200:
            out["conj"] = _close_approaches(a, op1, n, case["thresh"], _room(case)[2])
        return out
    # Propagated states: no 64-bit values apart from the propagator's own.
    return None
