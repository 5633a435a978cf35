"""Device buffers that grow together (csrc/wq3d_buffers.h, compiled here with
a counting allocator that fails at a chosen call): all are replaced, or the
old ones stay and nothing that was allocated on the way is kept.  A captured
graph holds the old addresses, so a failed growth must not release them."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "underseamodelinglibrary_b200", "csrc")

MAIN = r"""
#include <cstdio>
#include <set>
#include "wq3d_buffers.h"
int main() {
    for (int n = 1; n <= 4; ++n)
        for (int fail_at = 0; fail_at <= n; ++fail_at) {   /* n: no failure */
            std::set<void*> live;
            char pool[16];
            int next = 0, calls = 0;
            std::vector<wq3d::Resize> b;
            for (int k = 0; k < n; ++k) {
                void* p = k == 1 ? nullptr : &pool[next++];
                if (p) live.insert(p);
                b.push_back({p, (size_t)(100 + k), nullptr});
            }
            const std::set<void*> before = live;
            std::vector<size_t> sizes;
            const int rc = wq3d::make_all(
                b,
                [&](void** out, size_t bytes) {
                    if (calls++ == fail_at) return 7;
                    sizes.push_back(bytes);
                    *out = &pool[next++];
                    live.insert(*out);
                    return 0;
                },
                [&](void* p) {
                    if (!live.erase(p)) std::printf("released twice\n");
                });
            if (fail_at < n) {
                if (rc != 7 || live != before) std::printf("n %d fail %d: not restored\n", n, fail_at);
                for (auto& x : b)
                    if (x.fresh) std::printf("n %d fail %d: a new buffer is left\n", n, fail_at);
            } else {
                if (rc != 0 || (int)live.size() != (int)before.size() + n) std::printf("n %d: not made\n", n);
                for (int k = 0; k < n; ++k)
                    if (!live.count(b[k].fresh) || before.count(b[k].fresh) || sizes[k] != (size_t)(100 + k))
                        std::printf("n %d: buffer %d\n", n, k);
            }
        }
    std::printf("done\n");
    return 0;
}
"""


def test_all_or_none(tmp_path):
    (tmp_path / "main.cpp").write_text(MAIN)
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-Wall", "-Werror", "-I", CSRC, str(tmp_path / "main.cpp"),
                           "-o", str(tmp_path / "main")])
    assert subprocess.run([str(tmp_path / "main")], capture_output=True, text=True, check=True).stdout == "done\n"
