"""Room and warps for the CPA search's items (csrc/wq3d_targets.h, compiled
here).  A coarse fan's patches keep most targets: the list has room for every
patch and target that a small fan can leave, so that k_cpa is never left to
decide them one after another, and enough warps take them."""
import itertools
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "underseamodelinglibrary_b200", "csrc")

MAIN = r"""
#include <cstdio>
#include "wq3d_targets.h"
int main() {
    size_t nde, naz, nt, patches;
    while (std::scanf("%zu %zu %zu %zu", &nde, &naz, &nt, &patches) == 4)
        std::printf("%zu %zu %d\n", wq3d::cpa_patch_bound(nde, naz), wq3d::cpa_item_capacity(nde, naz, nt),
                    wq3d::cpa_item_blocks(nde * naz, patches, nt, 148));
    return 0;
}
"""


@pytest.fixture(scope="module")
def ask(tmp_path_factory):
    d = tmp_path_factory.mktemp("items")
    (d / "main.cpp").write_text(MAIN)
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-Wall", "-Werror", "-I", CSRC, str(d / "main.cpp"),
                           "-o", str(d / "main")])

    def call(rows):
        text = "\n".join("%d %d %d %d" % r for r in rows)
        out = subprocess.run([str(d / "main")], input=text, capture_output=True, text=True, check=True).stdout
        return [tuple(int(x) for x in line.split()) for line in out.splitlines()]

    return call


def _patches(nde, naz, shift):
    """every band of the fan cut the same way"""
    return -(-nde // (32 >> shift)) * -(-naz // (1 << shift))


def test_room_and_warps(ask):
    rows, most = [], []
    for nde, naz, nt in itertools.product((3, 7, 31, 32, 33, 69, 181, 907, 3601), (3, 8, 20, 33, 91, 181, 4096),
                                          (1, 32, 33, 1500, 4096, 100000)):
        p = max(_patches(nde, naz, s) for s in range(6))
        rows.append((nde, naz, nt, p))
        most.append(p)
    for (nde, naz, nt, p), (bound, room, blocks) in zip(rows, ask(rows)):
        assert bound == p
        assert 4096 <= room <= 1 << 20
        assert room >= min(p * nt, 1 << 18) and room >= min(2 * nde * naz, 1 << 20)
        assert 148 <= blocks <= 7 * 148
        # 16 items a warp, if 24 patches keep every target
        assert blocks == 7 * 148 or 4 * 16 * (blocks + 1) >= min(p, 24) * nt
        # a dense fan with few targets has a block for 256 rays
        assert 24 * nt > 64 * 148 or blocks == min(max(148, -(-nde * naz // 256)), 592)


def test_fans_that_used_to_overflow(ask):
    (_, room, blocks), = ask([(69, 8, 1500, 24)])
    assert room >= 24 * 1500 and blocks > 500
