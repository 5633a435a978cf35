"""The beam walks of k_eigenray take 15 cells of a side first with up to eight
frequencies and 32 with more.  A frequency's sum does not depend on the
others, nor on how the cells are taken: with one more, ninth, frequency above
them the first eight keep their bits.  Fans whose sides end around 14 to 16
and 30 to 34 cells and beyond, wrapping in AZ and not, and beams that end a
walk before and after."""
import numpy as np
import pytest

import underseamodelinglibrary_b200 as u
from underseamodelinglibrary_b200 import _abi
from underseamodelinglibrary_b200 import scenarios as S
from underseamodelinglibrary_b200 import types as T

pytestmark = pytest.mark.gpu


def _rays(nde, naz, wrap, f0, nf):
    T.compute_earth_radius(45.0)
    rng = np.random.default_rng(nde * 100 + naz)
    src = T.wposition1(45.0, -45.0, -300.0)
    tgt = T.wposition(1, 40, 45.0, -45.0, -100.0)
    for k in range(40):
        p = T.wposition1(src, float(rng.uniform(100.0, 4000.0)), float(rng.uniform(-0.1, 0.1)))
        tgt.latitude(0, k, p.latitude())
        tgt.longitude(0, k, p.longitude())
        tgt.altitude(0, k, -float(rng.uniform(1.0, 780.0)))
    ocean = u.ocean_model(u.boundary_flat(), u.boundary_flat(800.0, u.reflect_loss_rayleigh("sand")),
                          u.profile_linear(1500.0, 0.05))
    az = T.seq_linear(0.0, 360.0 / (naz - 1), naz) if wrap else T.seq_linear(-8.0, 16.0 / (naz - 1), naz)
    sc = dict(ocean=ocean, freq=T.seq_log(f0, 1.3, nf), pos=src, de=T.seq_linear(-40.0, 80.0 / (nde - 1), nde),
              az=az, dt=0.1, targets=tgt, type=_abi.HYBRID_GAUSSIAN, earth_radius=T.earth_radius())
    q = S.build_queue(sc, u.wave_queue)
    q.run(3.0)
    return q.take_eigenrays().arrays()


@pytest.mark.parametrize("f0", [30.0, 3000.0])
@pytest.mark.parametrize("nde,naz,wrap", [(18, 5, False), (31, 17, False), (33, 33, True), (35, 36, False),
                                          (67, 67, True), (180, 70, False)])
def test_frequencies_do_not_depend_on_one_another(engine, nde, naz, wrap, f0):
    few, more = _rays(nde, naz, wrap, f0, 8), _rays(nde, naz, wrap, f0, 9)
    assert len(few["time"]) > 10
    # a ninth frequency may bring an eigenray above the threshold; none is lost
    key = lambda a: list(zip(a["t2"], a["step"], a["de"], a["az"]))
    at = {k: n for n, k in enumerate(key(more))}
    rows = [at[k] for k in key(few)]
    for name in ("intensity", "phase"):
        assert np.array_equal(few[name], more[name][rows][:, :8]), name
    for name in ("time", "source_de", "source_az", "target_de", "target_az"):
        assert np.array_equal(few[name], more[name][rows]), name
