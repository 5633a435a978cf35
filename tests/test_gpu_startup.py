"""A queue's start-up follows the clearing of its counters and the upload of
its inputs: queues of a source so near the surface that rays reflect in the
very first step, made again and again, begin the same way every time."""
import hashlib

import pytest

import underseamodelinglibrary_b200 as u
from underseamodelinglibrary_b200 import _abi
from underseamodelinglibrary_b200 import scenarios as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("schedule", [_abi.REFLECT_SIDE, _abi.REFLECT_INLINE])
def test_first_steps_repeat(engine, schedule):
    scs = [S.gridded_munk(seed, 901, 45, 16, 1.0, src_depth=25.0) for seed in (1, 2)]
    seen = {}
    for k in range(240):
        sc = scs[k % 2]
        q = S.build_queue(sc, u.wave_queue, precision=_abi.FP32C)
        q.set_reflect_schedule(schedule)
        q.step(2)
        f = q.next()
        h = hashlib.sha1(f.rho.tobytes() + f.theta.tobytes() + f.surface.tobytes()).hexdigest()
        assert f.surface.sum() > 1000
        assert seen.setdefault(k % 2, h) == h, k
        del q


def _digest(sc):
    q = S.build_queue(sc, u.wave_queue, precision=_abi.FP32C)
    q.run(sc["time_max"])
    a = q.take_eigenrays().arrays()
    h = hashlib.sha1()
    for k in sorted(a):
        h.update(a[k].tobytes())
    return len(a["time"]), h.hexdigest()


def _fans():
    """one shape, three spacings of the rays (whose searches differ in
    length), and another shape"""
    from underseamodelinglibrary_b200 import types as T
    out = []
    for de in (T.seq_linear(-60.0, 1.0, 121), T.seq_linear(-6.0, 0.1, 121), T.seq_rayfan(-90.0, 90.0, 121)):
        sc = S.linear_slope_rayleigh(121, 19, 6, 7, 5.0)
        sc["de"] = de
        out.append(sc)
    out.append(S.linear_slope_rayleigh(61, 9, 3, 5, 5.0))
    return out


def test_reused_and_concurrent_queues_equal_fresh_ones(engine):
    """queues that take over a destroyed one's buffers, streams or memory, one
    after another and on four threads at once"""
    import threading
    scs = _fans()
    assert engine.wq3d_set_queue_cache(0) == 0
    fresh = [_digest(sc) for sc in scs]
    assert engine.wq3d_set_queue_cache(2) == 0
    assert [_digest(scs[k % 4]) for k in range(24)] == [fresh[k % 4] for k in range(24)]
    got = [None] * 4

    def work(t):
        got[t] = [_digest(scs[(t + k) % 4]) for k in range(8)]

    threads = [threading.Thread(target=work, args=(t,)) for t in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert got == [[fresh[(t + k) % 4] for k in range(8)] for t in range(4)]
    assert sum(n for n, _ in fresh) > 0


def test_memory_kept_between_queues_is_bounded_and_given_back(engine):
    import torch
    assert engine.wq3d_set_queue_cache(0) == 0
    torch.cuda.synchronize()
    free0, total = torch.cuda.mem_get_info()
    sc = S.reverb_scale(100.0, 901, 91, 64, 0.2)
    qs = [S.build_queue(sc, u.wave_queue, precision=_abi.FP32C) for _ in range(3)]
    del qs
    assert free0 - torch.cuda.mem_get_info()[0] <= total // 8 + (64 << 20)
    assert engine.wq3d_set_queue_cache(0) == 0
    assert free0 - torch.cuda.mem_get_info()[0] <= 64 << 20
    assert engine.wq3d_set_queue_cache(2) == 0
