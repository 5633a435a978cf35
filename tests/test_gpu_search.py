"""The CPA search against every pair: the bounds-checked build's FP64 form
takes every target of every patch of rays to the FP64 comparisons, and the
default build's eigenrays, in both forms, must equal its eigenrays bit for
bit.  Fans around the sizes where a patch or a band ends (3 rays, 31 to 34
rows, one AZ ray more or less than a patch holds), wrapping and not, with
steep and with narrow D/E; 1 to 20,000 targets around the sizes of a cluster
and of its shares, in a table's order and at random, above and below the
source (whose neighbours are compared by other rules), and more kept pairs
than the list holds."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = r"""
import hashlib, json, math, sys
import numpy as np
import underseamodelinglibrary_b200 as u
from underseamodelinglibrary_b200 import _abi, scenarios as S, types as T

def case(de, az, targets, seed, dt=0.1, time_max=4.0, depth=800.0, spreading=_abi.HYBRID_GAUSSIAN):
    T.compute_earth_radius(45.0)
    rng = np.random.default_rng(seed)
    src = T.wposition1(45.0, -45.0, -300.0)
    tgt = T.wposition(1, targets, 45.0, -45.0, -100.0)
    for k in range(targets):
        p = T.wposition1(src, float(rng.uniform(20.0, 5500.0)), float(rng.uniform(0.0, 2 * math.pi)))
        if k % 97 == 5:                      # above or below the source
            p = src
        tgt.latitude(0, k, p.latitude())
        tgt.longitude(0, k, p.longitude())
        tgt.altitude(0, k, -float(rng.uniform(1.0, depth)))
    ocean = u.ocean_model(u.boundary_flat(), u.boundary_flat(depth, u.reflect_loss_rayleigh("sand")),
                          u.profile_linear(1500.0, 0.05))
    return dict(ocean=ocean, freq=T.seq_log(1000.0, 2.0, 2), pos=src, de=de, az=az, dt=dt, targets=tgt,
                type=spreading, earth_radius=T.earth_radius()), time_max

def cases():
    L, F = T.seq_linear, T.seq_rayfan
    yield case(L(-60.0, 60.0, 3), L(-4.0, 4.0, 3), 1, 1)
    yield case(F(-90.0, 90.0, 31), L(0.0, 30.0, 13), 31, 2)
    yield case(F(-90.0, 90.0, 33), L(0.0, 30.0, 360.0), 32, 3)
    yield case(F(-90.0, 90.0, 34), L(10.0, 7.0, 32), 33, 4)
    yield case(L(-5.0, 0.1, 5.0), L(-10.0, 0.5, 33), 129, 5)
    yield case(F(-90.0, 90.0, 181), L(0.0, 4.0, 360.0), 700, 6)
    yield case(L(-89.0, 2.0, 89.0), L(0.0, 120.0, 360.0), 257, 7, spreading=_abi.CLASSIC_RAY)
    yield case(L(-80.0, 20.0, 9), L(-40.0, 16.0, 6), 20000, 8, time_max=2.0)
    sc = S.linear_slope_rayleigh(num_de=181, num_az=19, n_range=8, n_depth=9, time_max=9.0)
    yield sc, sc["time_max"]
    sc = S.gridded_munk(seed=5, num_de=121, num_az=13, n_targets=65, time_max=9.0, dt=0.05)
    yield sc, sc["time_max"]

def digest(sc, time_max, precision):
    q = S.build_queue(sc, u.wave_queue, precision=precision, eigenray_capacity=200000)
    q.run(time_max)
    a = q.take_eigenrays().arrays()
    h = hashlib.sha1()
    for k in sorted(a):
        h.update(np.ascontiguousarray(a[k]).tobytes())
    return [len(a["time"]), h.hexdigest()]

forms = [_abi.FP64] if _abi.LIB_PATH.endswith("checked.so") else [_abi.FP64, _abi.FP32C]
print(json.dumps([[digest(sc, t, f) for f in forms] for sc, t in cases()]))
"""


def _run(env_lib):
    env = dict(os.environ)
    env.pop("WQ3D_LIBRARY", None)
    if env_lib:
        env["WQ3D_LIBRARY"] = env_lib
    env["PYTHONPATH"] = ROOT + os.pathsep + env.get("PYTHONPATH", "")
    p = subprocess.run([sys.executable, "-c", SCRIPT], env=env, cwd=ROOT, capture_output=True, text=True, timeout=600)
    assert p.returncode == 0, p.stderr[-3000:]
    return json.loads(p.stdout.strip().splitlines()[-1])


def test_search_equals_every_pair(engine):
    every = _run("checked")
    plain = _run(None)
    assert len(every) == len(plain)
    for k, (e, p) in enumerate(zip(every, plain)):
        assert p[0] == e[0] and p[1] == e[0], (k, e, p)
    assert sum(e[0][0] for e in every) > 1000
