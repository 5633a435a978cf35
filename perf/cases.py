"""The workloads that this engine's speed is judged on, through its public
entry points: propagation of ray fans to eigenrays (analytic and gridded
oceans, every arithmetic form, small to large fans), batches of uneven
instances, reverberation (eigenverbs and bistatic eigenverbs) and the
gradient of transmission loss and travel time.

A case is a dict of plain values whose "family" names one of the functions
below.  ``prepare`` makes what a user's program holds before the call (ocean,
fan, targets, inputs); one ``run`` is the whole call: the queue is built, run
to its last step and its results are taken.  Sizes are those of the
repository's own scenarios and benchmark, and odd ones between them.
"""
import ctypes as C
import math

import numpy as np

import underseamodelinglibrary_b200 as u
from underseamodelinglibrary_b200 import _abi, adjoint
from underseamodelinglibrary_b200 import scenarios as S
from underseamodelinglibrary_b200 import types as T

FORMS = {"fp64": _abi.FP64, "fp32c": _abi.FP32C, "fp32": _abi.FP32}


def listed():
    return [
        # the smallest call: the reference's own three-path test scenario (25 x 9 rays, one target,
        # 35 steps), where building the queue and launching count for as much as the steps
        {"name": "basic_25x9", "family": "basic", "num_de": 25, "num_az": 9, "time_max": 3.5, "form": "fp64",
         "spreading": "gauss"},
        # monostatic reverberation of a small sonar: eigenverbs of 181 x 18 rays delivered to a
        # collection, then the bistatic overlap of that collection with itself
        {"name": "reverb_demo_181x18", "family": "reverb_demo", "num_de": 181, "num_az": 18, "time_max": 4.0},
        # the plain FP64 form in deep water: Munk profile, 100 targets, 600 steps
        {"name": "munk_fp64_181x37", "family": "munk", "num_de": 181, "num_az": 37, "targets": 10,
         "time_max": 60.0, "form": "fp64"},
        # the reference's published speed study: 3-D sound speed and bathymetry grids, 181 x 25 rays,
        # 100 targets, 801 steps, as one wavefront_generator task with its eigenray totals
        {"name": "std14_181x25", "family": "std14", "num_de": 181, "num_az": 25, "targets": 100,
         "time_max": 80.0, "form": "fp32c"},
        # one source in a gridded ocean with a middling fan
        {"name": "gridded_901x45", "family": "gridded", "num_de": 901, "num_az": 45, "targets": 64,
         "time_max": 30.0, "form": "fp32c"},
        # the headline workload: sloped bottom, 163,891 rays, 1024 targets, 5 frequencies, 801 steps
        {"name": "slope_1801x91", "family": "slope", "num_de": 1801, "num_az": 91, "ranges": 32, "depths": 32,
         "freqs": 5, "time_max": 40.0, "form": "fp32c"},
        # the same ocean in the plain FP64 form, with odd sizes throughout
        {"name": "slope_fp64_907x53", "family": "slope", "num_de": 907, "num_az": 53, "ranges": 23, "depths": 29,
         "freqs": 3, "time_max": 20.0, "form": "fp64"},
        # sixteen uneven sources and oceans advanced together on one GPU
        {"name": "batch_16", "family": "batch", "instances": 16, "max_de": 1801, "max_az": 91, "time_max": 30.0,
         "form": "fp32c"},
        # reverberation scale: 651,781 rays, 32 frequencies, 4096 targets, every eigenverb built
        # and counted
        {"name": "reverb_3601x181", "family": "reverb_scale", "num_de": 3601, "num_az": 181, "targets": 4096,
         "freqs": 32, "steps": 80, "form": "fp32c"},
        # forward and backward: TL and travel time at 64 receivers and their gradient with respect to
        # the sound speed profile and the bottom
        {"name": "gradient_901x45", "family": "gradient", "num_de": 901, "num_az": 45, "targets": 64,
         "steps": 800},
        # bistatic eigenverbs of two sensors, 57,600 footprints each
        {"name": "biverbs_57600", "family": "biverbs", "num_de": 160, "num_az": 360, "freqs": 2,
         "scattering": "constant"},
        # a short-range sonar's footprints: few, and more frequencies
        {"name": "biverbs_2700", "family": "biverbs", "num_de": 45, "num_az": 60, "freqs": 7,
         "scattering": "lambert"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["basic", "reverb_demo", "munk", "std14", "gridded", "slope", "slope", "batch",
                         "reverb_scale", "gradient", "biverbs"])
    if family == "basic":
        return {"family": family, "num_de": rng.randint(9, 61), "num_az": rng.randint(4, 25),
                "time_max": round(rng.uniform(2.5, 6.0), 2), "form": rng.choice(["fp64", "fp32c"]),
                "spreading": rng.choice(["gauss", "gauss", "classic"])}
    if family == "reverb_demo":
        return {"family": family, "num_de": rng.randint(61, 181), "num_az": rng.randint(6, 18),
                "time_max": round(rng.uniform(2.0, 4.0), 2)}
    if family == "munk":
        return {"family": family, "num_de": _log_int(rng, 37, 361), "num_az": _log_int(rng, 5, 73),
                "targets": rng.randint(2, 16), "time_max": round(rng.uniform(20.0, 60.0), 1),
                "form": rng.choice(["fp64", "fp64", "fp32c", "fp32"])}
    if family == "std14":
        return {"family": family, "num_de": _log_int(rng, 45, 361), "num_az": rng.choice([13, 25, 37, 49]),
                "targets": _log_int(rng, 1, 1000), "time_max": 80.0, "form": rng.choice(["fp64", "fp32c", "fp32c"])}
    if family == "gridded":
        return {"family": family, "num_de": _log_int(rng, 91, 1801), "num_az": _log_int(rng, 3, 91),
                "targets": _log_int(rng, 8, 256), "time_max": round(rng.uniform(10.0, 30.0), 1),
                "form": rng.choice(["fp64", "fp32c", "fp32c"])}
    if family == "slope":
        return {"family": family, "num_de": _log_int(rng, 91, 1801), "num_az": _log_int(rng, 7, 91),
                "ranges": rng.randint(3, 32), "depths": rng.randint(3, 32), "freqs": rng.randint(1, 8),
                "time_max": round(rng.uniform(10.0, 40.0), 1), "form": rng.choice(["fp64", "fp32c", "fp32c", "fp32"])}
    if family == "batch":
        return {"family": family, "instances": rng.randint(4, 16), "max_de": rng.randint(200, 1801),
                "max_az": rng.randint(7, 91), "time_max": round(rng.uniform(10.0, 30.0), 1),
                "form": rng.choice(["fp64", "fp32c", "fp32c"])}
    if family == "reverb_scale":
        return {"family": family, "num_de": _log_int(rng, 451, 3601), "num_az": _log_int(rng, 23, 181),
                "targets": _log_int(rng, 64, 4096), "freqs": rng.randint(3, 32), "steps": rng.randint(30, 80),
                "form": "fp32c"}
    if family == "gradient":
        return {"family": family, "num_de": _log_int(rng, 121, 901), "num_az": _log_int(rng, 9, 45),
                "targets": rng.randint(4, 64), "steps": rng.randint(200, 800)}
    return {"family": family, "num_de": _log_int(rng, 12, 160), "num_az": _log_int(rng, 18, 360),
            "freqs": rng.randint(1, 8), "scattering": rng.choice(["constant", "lambert", "chapman"])}


# ---------------------------------------------------------------- inputs
def _move_source(sc, rng, lo, hi):
    """the scenario's source at a random depth between lo and hi metres"""
    sc["pos"] = T.wposition1(sc["pos"].latitude(), sc["pos"].longitude(), -float(rng.uniform(lo, hi)))


def _freqs(n):
    """n log-spaced frequencies from 100 Hz, 3 kHz at most"""
    return T.seq_log(100.0, 30.0 ** (1.0 / max(n - 1, 4)), n)


def _basic(case, rng):
    sc = S.eigenray_basic()
    nde, naz = case["num_de"], case["num_az"]
    sc["de"] = T.seq_linear(-60.0, 120.0 / (nde - 1), nde)
    sc["az"] = T.seq_linear(-4.0, 8.0 / (naz - 1), naz)
    sc["time_max"] = case["time_max"]
    _move_source(sc, rng, 600.0, 1400.0)
    sc["targets"] = T.wposition(1, 1, 45.0 + float(rng.uniform(0.015, 0.025)), -45.0, -float(rng.uniform(600, 1400)))
    sc["type"] = _abi.CLASSIC_RAY if case["spreading"] == "classic" else _abi.HYBRID_GAUSSIAN
    return sc


def _munk(case, rng):
    sc = S.munk_flat(case["num_de"], case["num_az"], case["targets"], case["time_max"])
    _move_source(sc, rng, 700.0, 1500.0)
    return sc


def _near_targets(sc, rng, n, time):
    """n targets in the water that the fan crosses within a time"""
    sc["targets"] = S.random_targets(rng, sc["pos"], n, max_range=min(100e3, 1450.0 * time))


def _gridded(case, rng):
    sc = S.gridded_munk(int(rng.integers(1 << 31)), case["num_de"], case["num_az"], case["targets"],
                        case["time_max"], src_depth=float(rng.uniform(20.0, 500.0)))
    _near_targets(sc, rng, case["targets"], case["time_max"])
    return sc


def _slope(case, rng):
    sc = S.linear_slope_rayleigh(case["num_de"], case["num_az"], case["ranges"], case["depths"], case["time_max"])
    sc["freq"] = _freqs(case["freqs"])
    _move_source(sc, rng, 30.0, 100.0)
    return sc


def _batch(case, rng):
    scs = S.batched_gridded(case["instances"], int(rng.integers(1 << 31)), (91, case["max_de"]),
                            (1, case["max_az"]), (case["time_max"] / 3.0, case["time_max"]))
    for sc in scs:
        _near_targets(sc, rng, 64, sc["time_max"])
    return scs


def _reverb_scale(case, rng):
    sc = S.reverb_scale(float(rng.uniform(20.0, 800.0)), case["num_de"], case["num_az"], case["targets"],
                        (case["steps"] - 0.5) * 0.05, int(rng.integers(1 << 31)))
    sc["freq"] = T.seq_log(100.0, 100.0 ** (1.0 / 31.0), case["freqs"])
    _near_targets(sc, rng, case["targets"], case["steps"] * 0.05)
    return sc


def _rows(case):
    """rows of the tables that a pass fills with its eigenrays or biverbs"""
    family = case["family"]
    nt = {"basic": 1, "batch": 64 * case.get("instances", 0), "munk": case.get("targets", 0) ** 2}.get(
        family, case.get("targets", case.get("ranges", 1) * case.get("depths", 1)))
    if family == "biverbs":
        return 4 * case["num_de"] * case["num_az"]
    if family == "reverb_demo":
        return 64 * case["num_de"] * case["num_az"]
    return 64 + nt * {"reverb_scale": 24, "slope": 192}.get(family, 96)


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    family = case["family"]
    st = {"case": case, "form": FORMS[case.get("form", "fp64")]}
    rows, nf = _rows(case), case.get("freqs", 3 if family == "basic" else 1)
    if family == "biverbs":
        T.set_earth_radius(6371000.0)
        de = -85.0 + 80.0 / case["num_de"] * np.arange(case["num_de"])
        az = 360.0 / case["num_az"] * np.arange(case["num_az"])
        depth = float(rng.uniform(400.0, 600.0))
        st["src"] = S.analytic_footprints(0.0, 0.0, depth, de, az, case["freqs"])
        st["rcv"] = S.analytic_footprints(float(rng.uniform(0.004, 0.009)), float(rng.uniform(0.004, 0.009)), depth,
                                          de, az, case["freqs"])
        st["freq"] = 1000.0 * np.arange(1.0, case["freqs"] + 1.0)
        st["model"] = {"constant": u.scattering_constant(-30.0), "lambert": u.scattering_lambert(-27.0),
                       "chapman": u.scattering_chapman(10.0)}[case["scattering"]]
        st["out"] = (_abi.wq3d_biverb * rows)()
        st["power"] = np.zeros((rows, nf))
        return st
    if family == "gradient":
        st["sc"] = adjoint.AdjointScenario(case["num_de"], case["num_az"], case["steps"], case["targets"],
                                           seed=int(rng.integers(1 << 31)),
                                           max_range=min(50e3, 1400.0 * case["steps"] * 0.05))
        st["nodes"] = adjoint.munk_nodes(20, int(rng.integers(1 << 31)))
        st["w"] = rng.normal(size=(2, rows))
        st["table"] = {"values": np.zeros((rows, 2)), "d_bottom": np.zeros((rows, 3))}
        return st
    if family == "reverb_demo":
        st["sc"] = sc = S.eigenverb_demo()
        sc["ocean"] = u.ocean_model(u.boundary_flat(0.0, None, u.scattering_chapman(10.0)),
                                    u.boundary_flat(200.0, u.reflect_loss_rayleigh("sand"), u.scattering_lambert()),
                                    u.profile_linear(1500.0, u.attenuation_constant(0.0)))
        st["table"] = {k: [np.zeros((rows,) + shape) for _ in range(2)] for k, shape in
                       (("power", (1,)), ("time", ()), ("duration", ()))}
        st["table"]["index"] = [np.zeros((rows, 4), dtype=np.int64) for _ in range(2)]
        sc["de"] = T.seq_rayfan(-90.0, 90.0, case["num_de"])
        sc["az"] = T.seq_linear(0.0, 360.0 / case["num_az"], case["num_az"])
        sc["pos"] = T.wposition1(45.0, -45.0, -float(rng.uniform(5.0, 60.0)))
    elif family == "std14":
        st["sc"] = sc = S.std14(case["targets"], case["time_max"])
        sc["de"] = T.seq_rayfan(-90.0, 90.0, case["num_de"])
        sc["az"] = T.seq_linear(0.0, 360.0 / (case["num_az"] - 1), case["num_az"])
        _move_source(sc, rng, 100.0, 400.0)
    else:
        st["sc"] = {"basic": _basic, "munk": _munk, "gridded": _gridded, "slope": _slope, "batch": _batch,
                    "reverb_scale": _reverb_scale}[family](case, rng)
        st["table"] = {"values": np.zeros((rows, len(_COLUMNS))), "intensity": np.zeros((rows, nf)),
                       "phase": np.zeros((rows, nf)), "counts": np.zeros((rows, len(_COUNTS)), dtype=np.int64)}
    for sc in st["sc"] if family == "batch" else [st["sc"]]:
        T.set_earth_radius(sc["earth_radius"])
        sc["ocean"].handle()
    return st


# ---------------------------------------------------------------- one pass
_COLUMNS = ("time", "source_de", "source_az", "target_de", "target_az")
_COUNTS = ("surface", "bottom", "caustic", "upper", "lower", "t1", "t2", "de", "az", "step")


def _fill(table, rays, at=0):
    """an eigenray_list into rows of the program's table; returns the row after it"""
    a, end = rays.arrays(), at + len(rays)
    for j, k in enumerate(_COLUMNS):
        table["values"][at:end, j] = a[k]
    for j, k in enumerate(_COUNTS):
        table["counts"][at:end, j] = a[k]
    table["intensity"][at:end] = a["intensity"]
    table["phase"][at:end] = a["phase"]
    return end


def _generator(sc, form, listener, reverb):
    th = sc.get("thresholds", {})
    return u.wavefront_generator(sc["ocean"], sc["pos"], sc["targets"], None, sc["freq"], sc["de"], sc["az"],
                                 sc["dt"], sc["time_max"], compute_reverb=reverb, precision=form, listener=listener,
                                 **th)


def _run_reverb_demo(st):
    sc = st["sc"]
    T.set_earth_radius(sc["earth_radius"])
    gen = _generator(sc, st["form"], None, True)
    gen.run()
    verbs = gen.eigenverbs
    bv = u.biverb_generator(sc["ocean"], verbs, verbs, sc["freq"])
    bv.run()
    t, num = st["table"], []
    for k in range(2):
        num += [verbs.size(k), bv.collection().size(k)]
        if num[-1] == 0:
            continue
        rec, power = bv.collection().biverbs(k).arrays()
        n = len(rec)
        t["power"][k][:n] = power
        t["time"][k][:n] = rec["travel_time"]
        t["duration"][k][:n] = rec["duration"]
        for j, f in enumerate(("source", "receiver", "source_bottom", "receiver_surface")):
            t["index"][k][:n, j] = rec[f]
    return dict(t, num=num)


def _run_std14(st):
    sc = st["sc"]
    T.set_earth_radius(sc["earth_radius"])
    gen = _generator(sc, st["form"], None, False)
    gen.run()
    col = gen.eigenrays
    tot = [col.total(t, 0) for t in range(col.size1())]
    return {"num": col.num_eigenrays(),
            "values": np.array([[t.travel_time, t.source_de, t.source_az, t.target_de, t.target_az] for t in tot]),
            "intensity": np.array([t.intensity for t in tot]), "phase": np.array([t.phase for t in tot]),
            "counts": np.array([[t.surface, t.bottom, t.caustic, t.upper, t.lower] for t in tot])}


def _run_gradient(st):
    T.set_earth_radius(st["sc"].earth_radius)
    prop = adjoint.Propagation(st["sc"], st["nodes"], precision=_abi.FP32C)
    n = len(prop.eigenrays)
    g_nodes, g_bottom, _ = prop.vjp(st["w"][0, :n], st["w"][1, :n])
    st["table"]["values"][:n] = prop.values
    st["table"]["d_bottom"][:n] = prop.d_bottom
    return dict(st["table"], num=n, g_nodes=g_nodes, g_bottom=g_bottom)


def _run_biverbs(st):
    dp = C.POINTER(C.c_double)
    (s, sp), (r, rp) = st["src"], st["rcv"]
    lib = _abi.load_engine()
    desc = st["model"].desc()
    count = C.c_size_t()
    _abi.check(lib, lib.wq3d_biverbs(s, sp.ctypes.data_as(dp), len(sp), r, rp.ctypes.data_as(dp), len(rp),
                                     st["freq"].ctypes.data_as(dp), st["freq"].size, C.byref(desc), 6371000.0, 1.5,
                                     1e-20, st["out"], st["power"].ctypes.data_as(dp), len(st["out"]),
                                     C.byref(count)))
    rec = np.ctypeslib.as_array(st["out"])
    return {"power": st["power"], "time": rec["travel_time"], "duration": rec["duration"], "num": count.value,
            "source": rec["source"], "receiver": rec["receiver"]}


def run(st):
    family = st["case"]["family"]
    if family == "reverb_demo":
        return _run_reverb_demo(st)
    if family == "std14":
        return _run_std14(st)
    if family == "gradient":
        return _run_gradient(st)
    if family == "biverbs":
        return _run_biverbs(st)
    sc = st["sc"]
    if family == "batch":
        qs = [S.build_queue(s, u.wave_queue, precision=st["form"]) for s in sc]
        u.run_batch(qs, [s["time_max"] for s in sc])
        n = 0
        for q in qs:
            n = _fill(st["table"], q.take_eigenrays(), n)
        return dict(st["table"], num=n)
    q = S.build_queue(sc, u.wave_queue, precision=st["form"])
    if family == "reverb_scale":
        q.count_eigenverbs()
    q.run(sc["time_max"])
    out = dict(st["table"], num=_fill(st["table"], q.take_eigenrays()))
    if family == "reverb_scale":
        out["eigenverbs"] = np.array(q.eigenverb_counts())
    return out


# ---------------------------------------------------------------- work
def work(case):
    """FP64 operations of the ray steps themselves (about 130 per ray and
    step, plus 4 per frequency) without the eigenray search, which need not
    visit every ray and target; bytes are the inputs and the fronts' final
    state.  A footprint pair that overlaps costs about 200 operations, and
    about one pair in 50,000 does."""
    family = case["family"]
    if family == "biverbs":
        n = case["num_de"] * case["num_az"]
        rec, nf = 144, case["freqs"]
        return {"bytes": 2.0 * n * (rec + 8 * nf) + 1.1 * n * (104 + 8 * nf), "flops": 2.0 * n * 300 + 1.1 * n * 200}
    if family == "batch":
        rays, steps, nf, nt = case["instances"] * (91 + case["max_de"]) / 2 * (1 + case["max_az"]) / 2, \
            case["time_max"] * 2 / 3 / 0.05, 1, 64
    else:
        dt = {"basic": 0.1, "reverb_demo": 0.1, "munk": 0.1, "std14": 0.1, "gridded": 0.1}.get(family, 0.05)
        rays = float(case["num_de"] * case["num_az"])
        steps = case["steps"] if "steps" in case else case["time_max"] / dt
        nf, nt = case.get("freqs", 1), case.get("targets", case.get("ranges", 1) * case.get("depths", 1))
    gridded = family in ("std14", "gridded", "batch", "reverb_scale")
    passes = 10.0 if family == "gradient" else 1.0  # the forward, its recomputation and 8 directions back
    return {"bytes": rays * 8 * (18 + 2 * nf) + nt * 8.0 * (3 + nf),
            "flops": rays * steps * passes * ((400 if gridded else 130) + 4 * nf)}


# ---------------------------------------------------------------- 64-bit results
def _destination(lat, lng, rng, bearing):
    """the point at an angular range and bearing, in radians"""
    lat2 = np.arcsin(np.sin(lat) * np.cos(rng) + np.cos(lat) * np.sin(rng) * np.cos(bearing))
    lng2 = lng + np.arctan2(np.sin(bearing) * np.sin(rng) * np.cos(lat), np.cos(rng) - np.sin(lat) * np.sin(lat2))
    return np.degrees(lat2), np.degrees(lng2)


def _exact_biverbs(case, seed):
    """The overlap of two Gaussian footprints (one exponential of the offset
    in the receiver footprint's axes over the summed covariances) of every
    pair whose source centre lies inside the quadrilateral of half-diagonals
    1.5 length and 1.5 width around the receiver's."""
    st = prepare(case, seed)
    (s, sp), (r, rp) = st["src"], st["rcv"]
    s, r, R = np.ctypeslib.as_array(s), np.ctypeslib.as_array(r), 6371000.0
    slat, slng = 90.0 - np.degrees(s["position"][:, 1]), np.degrees(s["position"][:, 2])
    rlat, rlng = np.pi / 2 - r["position"][:, 1], r["position"][:, 2]
    corners = [_destination(rlat, rlng, 1.5 * (r["length"] if k % 2 == 0 else r["width"]) / r["position"][:, 0],
                            r["direction"] + k * np.pi / 2) for k in range(4)]
    cx, cy = np.stack([c[0] for c in corners]), np.stack([c[1] for c in corners])
    order = np.argsort(slat, kind="stable")
    lo = np.searchsorted(slat[order], cx.min(0), "right")
    hi = np.searchsorted(slat[order], cx.max(0), "left")
    si, ri = [], []
    for j in range(len(r)):
        c = order[lo[j]:hi[j]]
        c = c[(slng[c] > cy[:, j].min()) & (slng[c] < cy[:, j].max())]
        if c.size == 0:
            continue
        x, y = slat[c], slng[c]
        e = [(cx[(k + 1) % 4, j] - cx[k, j]) * (y - cy[k, j]) - (cy[(k + 1) % 4, j] - cy[k, j]) * (x - cx[k, j])
             for k in range(4)]
        c = np.sort(c[np.all(np.array(e) > 0, axis=0) | np.all(np.array(e) < 0, axis=0)])
        si.append(c)
        ri.append(np.full(c.size, j))
    si, ri = np.concatenate(si), np.concatenate(ri)
    a, b = s[si], r[ri]
    lat1, lng1, lat2, lng2 = rlat[ri], rlng[ri], np.pi / 2 - a["position"][:, 1], a["position"][:, 2]
    arc = 2 * np.arcsin(np.sqrt(np.sin(0.5 * (lat1 - lat2)) ** 2
                                + np.cos(lat1) * np.cos(lat2) * np.sin(0.5 * (lng1 - lng2)) ** 2))
    az = np.arctan2(np.sin(lng1 - lng2) * np.cos(lat2),
                    np.cos(lat1) * np.sin(lat2) - np.sin(lat1) * np.cos(lat2) * np.cos(lng1 - lng2))
    az = np.where((np.abs(arc) < 1e-6) | (np.abs(lat1) < 1e-10), np.where(lat1 > 0, np.pi, 0.0),
                  np.fmod(2 * np.pi - az, 2 * np.pi))
    dist = arc * b["position"][:, 0]
    az = np.where(dist < 1e-6, 0.0, az) - b["direction"]
    y2, x2 = (dist * np.cos(az)) ** 2, (dist * np.sin(az)) ** 2
    two = 2 * (a["direction"] - b["direction"])
    sl, sw, rl, rw = a["length"] ** 2, a["width"] ** 2, b["length"] ** 2, b["width"] ** 2
    det = 0.5 * (2 * (sl * sw + rl * rw) + (sl + sw) * (rl + rw) - (sl - sw) * (rl - rw) * np.cos(two))
    kappa = -0.25 * (x2 * (sl + sw + (sl - sw) * np.cos(two) + 2 * rl)
                     + y2 * (sl + sw - (sl - sw) * np.cos(two) + 2 * rw)
                     - 2 * np.sqrt(x2 * y2) * (sl - sw) * np.sin(two)) / det
    sigma = 0.5 * ((1 / sw + 1 / sl) + (1 / sw - 1 / sl) * np.cos(two) + 2 / rw) / (det / (sl * sw * rl * rw))
    gs, gr = a["grazing"][:, None], b["grazing"][:, None]
    if case["scattering"] == "lambert":
        strength = 10.0 ** -2.7 * np.abs(np.sin(gs) * np.sin(gr))
    elif case["scattering"] == "constant":
        strength = 10.0 ** -3.0
    else:
        return None
    power = 0.125 * sp[si] * rp[ri] * strength * (np.exp(kappa) / np.sqrt(det))[:, None]
    keep = power.max(axis=1) >= 1e-20
    duration = 0.5 * np.cos(b["grazing"]) / b["sound_speed"] * np.sqrt(sigma)

    def table(v):
        out = np.zeros((_rows(case),) + v.shape[1:])
        out[:keep.sum()] = v[keep]
        return out

    return {"power": table(power), "time": table(a["travel_time"] + b["travel_time"]), "duration": table(duration),
            "num": None, "source": None, "receiver": None}


def exact(case, seed):
    """Footprint overlaps have a closed form; eigenrays are what a chain of
    finite steps, searches and thresholds finds, and have none."""
    return _exact_biverbs(case, seed) if case["family"] == "biverbs" else None
