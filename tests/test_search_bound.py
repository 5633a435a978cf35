"""The bounds of the CPA search (feature_diff, set_range, target_keeps and
cluster_keeps in csrc/wq3d_kernels.cu) restated in numpy: single precision
with one rounding per operation (a fused multiply-add rounds once), from
double coordinate differences.  A target or a cluster of targets that a
bound rejects must be rejected for every ray of the patch by the reference's
double expression, whose own rounding is 5 x 2^-53 (rho^2 + R^2) a point."""
import numpy as np

f = np.float32
U = f(5.9604645e-8)
R0 = 6.367e6


def fma(a, b, c):
    return (np.float64(a) * np.float64(b) + np.float64(c)).astype(f)


def features(other, own, ref):
    """[7, rays] single, and the theta and phi differences"""
    (ro, to, po), (r, t, p) = other, own
    rr, x, y = (f(r - ref[0]), f(t - ref[1]), f(p - ref[2]))
    dr, ds = f(ro - r), f(ro * np.sin(to) - r * np.sin(t))
    tx, ty, R, S = f(to - t), f(po - p), f(ro), f(ro * np.sin(to))
    two = f(2.0)
    d = [dr * fma(two, rr, dr), dr, fma(R * tx, fma(two, x, tx), x * x * dr), fma(R, tx, x * dr),
         fma(S * ty, fma(two, y, ty), y * y * ds), fma(S, ty, y * ds), ds]
    return np.stack(d).astype(f), tx, ty, np.abs(rr).max(), np.abs(x).max(), np.abs(y).max()


def weights(R, RS, Rr, X, Y):
    return np.stack([np.ones_like(R), R * X * X - 2.0 * Rr, R, -2.0 * R * X, RS, -2.0 * RS * Y, RS * Y * Y]).astype(f)


def ranges(d, tx, ty, W, rm, xm, ym):
    lo, hi = d.min(axis=1), d.max(axis=1)
    m = f(0.5) * (lo + hi)
    h = f(1.000001) * np.maximum(hi - m, m - lo)
    dxm, dym = np.abs(tx).max(), np.abs(ty).max()
    drm, dsm = abs(m[1]) + h[1], abs(m[6]) + h[6]
    two, g = f(2.0), drm * fma(f(2.0), rm, drm)
    g = fma(W[1], drm, g)
    g = fma(W[2], two * W[2] * dxm * fma(two, xm, dxm) + xm * xm * drm, g)
    g = fma(W[3], two * W[2] * dxm + xm * drm, g)
    g = fma(W[4], two * W[2] * dym * fma(two, ym, dym) + ym * ym * dsm, g)
    g = fma(W[5], two * W[2] * dym + ym * dsm, g)
    return m, h, fma(W[6], dsm, g)


def bound(w, m, h):
    a, b = f(m[0] + h[0]) * np.ones(w.shape[1], f), np.zeros(w.shape[1], f)
    for k in range(1, 7):
        a, b = fma(w[k], m[k], a), fma(np.abs(w[k]), h[k], b)
    return a + b


def distance2(p, t):
    """the reference's expression in extended precision"""
    L = np.longdouble
    a, b = (L(p[1]) - L(t[1])) / 2, (L(p[2]) - L(t[2])) / 2
    inner = 1 - 2 * (a * a + np.sin(L(t[1])) * np.sin(L(p[1])) * b * b)
    return L(p[0]) ** 2 + L(t[0]) ** 2 - 2 * L(t[0]) * L(p[0]) * inner


def test_bounds_reject_only_what_the_comparisons_reject():
    rng = np.random.default_rng(20261205)
    n_target = n_cluster = 0
    for _ in range(400):
        # a patch of 32 rays of some extent, and the point each is compared with
        size, step = 10.0 ** rng.uniform(0.0, 4.5), 10.0 ** rng.uniform(-1.0, 3.0)
        base = np.array([R0 - rng.uniform(0, 4000), rng.uniform(0.3, 2.5), rng.uniform(-3, 3)])
        met = np.array([1.0, 1.0 / R0, 1.0 / R0])
        own = base[:, None] + met[:, None] * size * rng.uniform(-1, 1, (3, 32)) * [[0.2], [1.0], [1.0]]
        u = rng.normal(size=3)
        u /= np.linalg.norm(u)
        other = own + met[:, None] * (step * u[:, None] + 0.05 * step * rng.normal(size=(3, 32)))
        ref = own[:, 16]
        # clusters of 32 targets close to the plane where the two distances are equal
        ncl, reach, spread = 8, 10.0 ** rng.uniform(2.0, 5.0), 10.0 ** rng.uniform(0.0, 3.0)
        off = rng.normal(size=(3, ncl)) * reach
        off -= u[:, None] * (u @ off) + u[:, None] * rng.uniform(-4, 8, ncl) * (size * rng.uniform(0, 1.5) + step)
        tgt = ref[:, None, None] + met[:, None, None] * (off[:, :, None] + spread * rng.normal(size=(3, ncl, 32)))
        t = tgt.reshape(3, -1)
        box = [t.min(axis=1), t.max(axis=1)]
        Xm, Ym, Rm = (f(max(abs(box[0][k] - ref[k]), abs(box[1][k] - ref[k]))) for k in (1, 2, 0))
        R = f(1.0001) * max(f(box[1][0]), f(ref[0]))
        W = [f(0), f(1.0001) * (R * Xm * Xm + f(2) * Rm), R, f(2) * R * Xm, R, f(2) * R * Ym, f(1.0001) * R * Ym * Ym]
        c0 = max(f(1), f(4e-15) * (f(ref[0]) * f(ref[0]) + R * R))
        d, tx, ty, rm, xm, ym = features(other, own, ref)
        m, h, g = ranges(d, tx, ty, W, rm, xm, ym)
        w = weights(t[0], t[0] * np.sin(t[1]), t[0] - ref[0], t[1] - ref[1], t[2] - ref[2])
        rejected = bound(w, m, h) + fma(f(96) * U, g, f(1.001) * c0) < 0
        true = distance2(other[:, :, None], t[:, None, :]) - distance2(own[:, :, None], t[:, None, :])
        worst = true.max(axis=0) + 2 * 5 * 2.0 ** -53 * (own[0].max() ** 2 + t[0] ** 2)
        assert np.all(worst[rejected] < 0)
        n_target += int(rejected.sum())
        # the clusters
        S = tgt[0] * np.sin(tgt[1])
        v = np.stack([tgt[0], tgt[1], tgt[2], S])
        mid = 0.5 * (v.min(axis=2) + v.max(axis=2))
        half = (np.maximum(v.max(axis=2) - mid, mid - v.min(axis=2)) * 1.000001).astype(f)
        dR, dT, dP, dS = half
        cw = weights(mid[0], mid[3], mid[0] - ref[0], mid[1] - ref[1], mid[2] - ref[2])
        ax, ay = np.abs(f(mid[1] - ref[1])), np.abs(f(mid[2] - ref[2]))
        Rt, St, two = cw[2] + dR, np.abs(cw[4]) + dS, f(2.0)
        D = [None, fma(two, dR, fma(Rt * dT, fma(two, ax, dT), ax * ax * dR)), dR, two * fma(Rt, dT, ax * dR), dS,
             two * fma(St, dP, ay * dS), fma(St * dP, fma(two, ay, dP), ay * ay * dS)]
        b = np.zeros(ncl, f)
        for k in range(1, 7):
            b = fma(D[k], abs(m[k]) + h[k], b)
        cut = fma(f(1.001), b, bound(cw, m, h)) + fma(f(192) * U, g, f(1.001) * c0) < 0
        assert np.all(worst.reshape(ncl, 32)[cut] < 0)
        n_cluster += int(cut.sum())
    assert n_target > 5000 and n_cluster > 100
