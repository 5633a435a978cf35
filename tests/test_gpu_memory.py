"""Queues with eigenverbs on a device whose memory is nearly all taken: record
buffers that grow stay within what is really free, whatever dropped queues
left behind, and every eigenverb is counted all the same."""
import pytest

import underseamodelinglibrary_b200 as u
from underseamodelinglibrary_b200 import _abi
from underseamodelinglibrary_b200 import scenarios as S

pytestmark = pytest.mark.gpu


def _counts(shapes):
    qs = []
    for nde, naz in shapes:
        sc = S.linear_slope_rayleigh(nde, naz, 4, 4, 4.0)
        q = S.build_queue(sc, u.wave_queue, precision=_abi.FP32C)
        q.count_eigenverbs(True)
        qs.append(q)
    u.run_batch(qs, 4.0)
    return [tuple(q.eigenverb_counts()) for q in qs]


@pytest.mark.parametrize("left_gb", [2.0, 4.0])
def test_eigenverbs_with_little_memory_left(engine, left_gb):
    import torch
    shapes = [(301, 31), (901, 61), (601, 41), (901, 61)]
    assert engine.wq3d_set_queue_cache(0) == 0
    hold = None
    try:
        want = _counts(shapes)
        assert all(sum(w) > 1000 for w in want)
        assert engine.wq3d_set_queue_cache(0) == 0
        engine.wq3d_set_queue_cache(2)
        free, _ = torch.cuda.mem_get_info()
        hold = torch.empty(max(1, int(free - left_gb * 2 ** 30)), dtype=torch.uint8, device="cuda")
        for order in (shapes, shapes[::-1], shapes):
            got = dict(zip(order, _counts(order)))
            assert got == dict(zip(shapes, want))
    finally:
        del hold
        torch.cuda.empty_cache()
        engine.wq3d_set_queue_cache(2)
