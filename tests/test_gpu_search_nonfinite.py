"""A target table in which some targets have NaN or infinite coordinates:
those get no eigenray, and every other target's eigenrays are those of the
table in which all are finite, bit for bit, in both forms.  The fan has more
interior rays than the candidate list has room for, and the bad target stands
first, in the middle and last of a cluster of 32, alone and among others."""
import math

import numpy as np
import pytest

import underseamodelinglibrary_b200 as u
from underseamodelinglibrary_b200 import _abi
from underseamodelinglibrary_b200 import scenarios as S
from underseamodelinglibrary_b200 import types as T

pytestmark = pytest.mark.gpu


def _scenario(nt):
    T.compute_earth_radius(45.0)
    rng = np.random.default_rng(nt)
    src = T.wposition1(45.0, -45.0, -300.0)
    tgt = T.wposition(1, nt, 45.0, -45.0, -100.0)
    for k in range(nt):
        p = T.wposition1(src, float(rng.uniform(20.0, 4000.0)), float(rng.uniform(0.0, 2 * math.pi)))
        tgt.latitude(0, k, p.latitude())
        tgt.longitude(0, k, p.longitude())
        tgt.altitude(0, k, -float(rng.uniform(1.0, 800.0)))
    ocean = u.ocean_model(u.boundary_flat(), u.boundary_flat(800.0, u.reflect_loss_rayleigh("sand")),
                          u.profile_linear(1500.0, 0.05))
    return dict(ocean=ocean, freq=T.seq_log(1000.0, 2.0, 2), pos=src, de=T.seq_rayfan(-90.0, 90.0, 91),
                az=T.seq_linear(0.0, 6.0, 360.0), dt=0.1, targets=tgt, type=_abi.HYBRID_GAUSSIAN,
                earth_radius=T.earth_radius())


def _run(sc, precision):
    q = S.build_queue(sc, u.wave_queue, precision=precision)
    q.run(3.0)
    return q.take_eigenrays().arrays()


@pytest.mark.parametrize("precision", [_abi.FP64, _abi.FP32C])
@pytest.mark.parametrize("nt", [2, 100])
def test_other_targets_keep_their_eigenrays(engine, nt, precision):
    sc = _scenario(nt)
    want = _run(sc, precision)
    assert len(want["time"]) > 0
    good = [sc["targets"].rho.copy(), sc["targets"].theta.copy(), sc["targets"].phi.copy()]
    for value in (math.nan, math.inf, -math.inf):
        for bad in sorted({0, nt // 2, min(31, nt - 1), nt - 1}):
            for rows in ([0], [1], [2], [0, 1, 2]):
                c = [x.copy() for x in good]
                for r in rows:
                    c[r][0, bad] = value
                sc["targets"].rho, sc["targets"].theta, sc["targets"].phi = c
                got = _run(sc, precision)
                keep = want["t2"] != bad
                assert not (got["t2"] == bad).any()
                for name in want:
                    assert np.array_equal(got[name], want[name][keep]), (value, bad, rows, name)


def test_no_finite_target(engine):
    sc = _scenario(3)
    sc["targets"].rho[:] = math.nan
    assert len(_run(sc, _abi.FP64)["time"]) == 0
