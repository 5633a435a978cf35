"""Grid interpolation on the GPU equals the oracle's bit for bit.

Interpolation is made of additions, multiplications and divisions, each of
which rounds to nearest on both sides, so no tolerance is needed.  The
device divides without branches and from tables, in unrolled forms per
dimension and kind; the sizes here are the smallest axes that each form
takes, cells with and without neighbours at both ends, equal and
alternating data (zero and sign-changing slopes), NaN data, points on the
nodes, beside them, beyond the ends and spread over many random spacings,
and magnitudes that send a grid to the general form."""
import ctypes as C

import numpy as np
import pytest

import underseamodelinglibrary_b200 as u
from underseamodelinglibrary_b200 import _abi
from oracle_binding import load_oracle

pytestmark = pytest.mark.gpu

LINEAR, PCHIP = u.data_grid.LINEAR, u.data_grid.PCHIP


def _oracle_speed(oc, R, rho, th, ph):
    od = oc.descriptor()
    c, g = np.empty(rho.size), np.empty(3 * rho.size)
    assert load_oracle().oracle_sound_speed(C.byref(od), R, rho.size, _abi.as_dp(rho), _abi.as_dp(th),
                                            _abi.as_dp(ph), _abi.as_dp(c), _abi.as_dp(g)) == 0
    return c, g.reshape(3, -1)


def _axis(rng, kind, n, x0, step):
    if kind == "linear":
        return u.seq_linear(x0, step, n)
    return u.seq_data(x0 + np.sign(step) * np.cumsum(abs(step) * rng.uniform(0.2, 1.8, n)))


def _points(rng, ax, n):
    """n points of an axis: nodes, their neighbours in rounding, the ends and beyond, and random ones"""
    x = np.asarray(ax.data)
    span = x[-1] - x[0]
    near = np.concatenate([x, np.nextafter(x, np.inf), np.nextafter(x, -np.inf), x[:1] - 0.3 * span, x[-1:] + 0.3 * span])
    return rng.permutation(np.concatenate([near, x[0] + span * rng.uniform(-0.05, 1.05, n)])[:n])


def _data(rng, shape, form, scale):
    d = 1500.0 + rng.normal(0.0, 20.0, shape)
    if form == "flat":
        d = np.round(d / 25.0) * 25.0          # runs of equal values
    elif form == "zigzag":
        d = 1500.0 + 5.0 * (np.indices(shape).sum(axis=0) % 2)
    elif form == "nan":
        d[tuple(s // 2 for s in shape)] = np.nan
    return d * scale


@pytest.mark.parametrize("sizes", [(2,), (4,), (5,), (33,), (2, 2), (4, 3), (17, 5), (2, 2, 2), (4, 2, 3), (5, 4, 2),
                                   (50, 20, 20)])
@pytest.mark.parametrize("form,scale", [("random", 1.0), ("flat", 1.0), ("zigzag", 1.0), ("nan", 1.0),
                                        ("random", 1e-30)])
def test_speed_and_gradient_bits(engine, sizes, form, scale):
    u.compute_earth_radius(45.0)
    R = u.earth_radius()
    rng = np.random.default_rng([len(sizes), *sizes, len(form)])
    npts = 3000
    for kinds in (("linear",) * 3, ("data",) * 3, ("data", "linear", "data")):
        for sign in (-1.0, 1.0):
            first = R if sign < 0 else R - 5000.0
            axes = [_axis(rng, kinds[0], sizes[0], first, sign * 5000.0 / max(sizes[0] - 1, 1))]
            axes += [_axis(rng, kinds[d], sizes[d], (0.7, -0.9)[d - 1], 0.03 / sizes[d]) for d in range(1, len(sizes))]
            pts = [np.ascontiguousarray(_points(rng, a, npts)) for a in axes]
            pts += [np.zeros(npts)] * (3 - len(pts))
            for k0 in (LINEAR, PCHIP):
                for edge in (True, False):
                    g = u.data_grid(axes, _data(rng, sizes, form, scale))
                    g.interp_type(0, k0)
                    for d in range(len(sizes)):
                        g.edge_limit(d, edge)
                    oc = u.ocean_model(u.boundary_flat(), u.boundary_flat(6000.0), u.profile_grid(g))
                    c, grad = oc.sound_speed(*pts)
                    co, go = _oracle_speed(oc, R, *pts)
                    np.testing.assert_array_equal(c, co)
                    np.testing.assert_array_equal(np.asarray(grad)[:len(sizes)], go[:len(sizes)])


def test_many_spacings(engine):
    """a division by each of 2,000 random spacings, 200,000 points"""
    u.compute_earth_radius(45.0)
    R = u.earth_radius()
    rng = np.random.default_rng(5)
    ax = _axis(rng, "data", 2000, R - 5000.0, 2.5)
    rho = rng.uniform(float(np.min(ax.data)), float(np.max(ax.data)), 200000)
    z = np.zeros(rho.size)
    for k0 in (LINEAR, PCHIP):
        g = u.data_grid([ax], rng.normal(1500.0, 10.0, 2000))
        g.interp_type(0, k0)
        oc = u.ocean_model(u.boundary_flat(), u.boundary_flat(6000.0), u.profile_grid(g))
        c, grad = oc.sound_speed(rho, z, z)
        co, go = _oracle_speed(oc, R, rho, z, z)
        np.testing.assert_array_equal(c, co)
        np.testing.assert_array_equal(np.asarray(grad)[0], go[0])
