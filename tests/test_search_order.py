"""The order in which cpa_targets (csrc/wq3d_targets.h, compiled here) takes
random targets is that of their Morton keys, equal keys in the caller's
order."""
import math
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
    if (std::scanf("%zu", &nt) != 1) return 1;
    std::vector<double> r(nt), th(nt), ph(nt), sn(nt);
    std::vector<uint8_t> branch(nt);
    for (size_t t = 0; t < nt; ++t) {
        if (std::scanf("%la %la %la %la", &r[t], &th[t], &ph[t], &sn[t]) != 4) return 1;
    }
    wq3d::CpaTargets o;
    wq3d::cpa_targets(r, th, ph, sn, branch, &o);
    for (uint32_t i : o.index) std::printf("%u ", i);
    return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("order")
    (d / "main.cpp").write_text(MAIN)
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-Wall", "-Werror", "-I", CSRC, str(d / "main.cpp"),
                           "-o", str(d / "main")])
    return str(d / "main")


@pytest.mark.parametrize("nt,grid", [(100, 0), (200, 0), (1000, 5), (5000, 0), (5000, 40)])
def test_morton_order(program, nt, grid):
    rng = np.random.default_rng(nt + grid)
    u = rng.uniform(0.0, 1.0, (3, nt))
    if grid:
        u = np.floor(u * grid) / grid  # many equal keys
    bad = nt // 3
    r, th, ph = 6.37e6 - 4000.0 * u[0], 0.78 + 0.01 * u[1], -0.9 + 0.01 * u[2]
    r[bad] = math.nan
    sn = [math.sin(x) for x in th]
    text = "%d\n" % nt + "\n".join("%s %s %s %s" % tuple(float(x).hex() if x == x else "nan" for x in row)
                                   for row in zip(r, th, ph, sn))
    got = [int(x) for x in subprocess.run([program], input=text, capture_output=True, text=True,
                                          check=True).stdout.split()]
    good = [t for t in range(nt) if t != bad]
    lo = [min(float(a[t]) for t in good) for a in (r, th, ph)]
    hi = [max(float(a[t]) for t in good) for a in (r, th, ph)]
    size = max(hi[0] - lo[0], hi[0] * (hi[1] - lo[1]), hi[0] * (hi[2] - lo[2]))

    def key(t):
        x = (float(r[t]) - lo[0], hi[0] * (float(th[t]) - lo[1]), hi[0] * sn[t] * (float(ph[t]) - lo[2]))
        c = [int(min(1023.0, max(0.0, 1023.0 * v / size))) for v in x]
        return sum(((c[k] >> b) & 1) << (3 * b + k) for b in range(10) for k in range(3))

    assert got == sorted(good, key=lambda t: (key(t), t))
