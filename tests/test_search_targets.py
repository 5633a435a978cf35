"""The clusters of targets that the CPA search trusts (csrc/wq3d_targets.h,
compiled here): every target with finite coordinates is in exactly one
cluster, lies within that cluster's extents and within the box, and a target
with a NaN or infinite coordinate, wherever it stands, is in none."""
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "underseamodelinglibrary_b200", "csrc")

MAIN = r"""
#include <cstdio>
#include "wq3d_targets.h"
int main() {
    size_t nt;
    while (std::scanf("%zu", &nt) == 1) {
        std::vector<double> r(nt), th(nt), ph(nt), sn(nt);
        std::vector<uint8_t> branch(nt);
        for (size_t t = 0; t < nt; ++t) {
            if (std::scanf("%lf %lf %lf", &r[t], &th[t], &ph[t]) != 3) return 1;
            sn[t] = std::sin(th[t]);
        }
        wq3d::CpaTargets o;
        wq3d::cpa_targets(r, th, ph, sn, branch, &o);
        std::printf("%zu %zu\n", o.index.size(), o.clusters.size());
        for (double b : o.box) std::printf("%.17g ", b);
        for (uint32_t i : o.index) std::printf("%u ", i);
        for (double v : o.tgt) std::printf("%.17g ", v);
        for (const wq3d::TgtCluster& c : o.clusters)
            std::printf("%.17g %.17g %.17g %.17g %.17g %.17g %.17g %.17g ", c.R, c.T, c.P, c.RS, (double)c.dR,
                        (double)c.dT, (double)c.dP, (double)c.dRS);
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("targets")
    (d / "main.cpp").write_text(MAIN)
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-Wall", "-Werror", "-I", CSRC, str(d / "main.cpp"),
                           "-o", str(d / "main")])
    return str(d / "main")


def _tables():
    rng = np.random.default_rng(1)
    for nt in (1, 5, 32, 33, 100, 700):
        t = np.stack([6.37e6 - rng.uniform(1.0, 5000.0, nt), rng.uniform(0.7, 0.8, nt), rng.uniform(-1.0, -0.9, nt)])
        yield t
        for value in (np.nan, np.inf, -np.inf):
            for k in (0, min(nt - 1, 17), nt - 1):
                for rows in ([0], [1], [2], [0, 1, 2]):
                    bad = t.copy()
                    bad[rows, k] = value
                    yield bad
        bad = t.copy()
        bad[rng.integers(0, 3, nt), np.arange(nt)] = np.nan
        yield bad


def test_clusters_hold_their_targets(program):
    tables = list(_tables())
    text = "".join("%d\n%s\n" % (t.shape[1], " ".join("%.17g" % v for v in t.T.ravel())) for t in tables)
    v = iter(subprocess.run([program], input=text, capture_output=True, text=True, check=True).stdout.split())

    def take(n):
        return np.array([float(next(v)) for _ in range(n)])

    for t in tables:
        finite = np.flatnonzero(np.isfinite(t).all(axis=0))
        n, ncl = (int(x) for x in take(2))
        box, index = take(6), take(n).astype(int)
        tgt, cl = take(4 * n).reshape(n, 4), take(8 * ncl).reshape(ncl, 8)
        assert sorted(index) == list(finite) and ncl == (n + 31) // 32
        t = np.where(np.isfinite(t), t, 0.0)
        want = np.stack([t[0], t[1], t[2], np.sin(t[1])], axis=1)[index] if n else np.zeros((0, 4))
        assert np.array_equal(tgt[:, :3], want[:, :3]) and np.allclose(tgt[:, 3], want[:, 3], rtol=1e-15)
        if n:
            assert np.array_equal(box[0::2], tgt[:, :3].min(axis=0)) and np.array_equal(box[1::2], tgt[:, :3].max(axis=0))
        at = np.concatenate([tgt[:, :3], tgt[:, :1] * tgt[:, 3:]], axis=1)
        for j in range(n):
            c = cl[j // 32]
            assert np.all(np.abs(at[j] - c[:4]) <= c[4:]), (j, at[j], c)
