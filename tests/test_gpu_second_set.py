"""A queue whose second set of result buffers, which only lets the host copy
one chunk while the next runs, finds no room: the queue is made and computes
the same, the destroyed queues kept for reuse stay, and no error text is left."""
import numpy as np
import pytest

import underseamodelinglibrary_b200 as u
from underseamodelinglibrary_b200 import scenarios as S
from underseamodelinglibrary_b200 import types as T

pytestmark = pytest.mark.gpu

GB = 1 << 30


def _queue(nf):
    """records of nf frequencies: 2^21 of them a result set, 0.47 GB at 8
    frequencies and 2.35 GB at 64"""
    sc = S.eigenray_basic()
    sc["freq"] = T.seq_log(1000.0, 1.05, nf)
    q = S.build_queue(sc, u.wave_queue, eigenray_capacity=1 << 17)
    return q, sc


def _rays(q, sc):
    q.run(sc["time_max"])
    r = q.take_eigenrays()
    return r.arrays()


def test_second_result_set_without_room(engine):
    import torch
    hold = None
    try:
        assert engine.wq3d_set_queue_cache(0) == 0
        q, sc = _queue(64)
        want = _rays(q, sc)
        assert len(want["time"]) > 0
        del q
        assert engine.wq3d_set_queue_cache(0) == 0  # gives its memory back
        assert engine.wq3d_set_queue_cache(2) == 0
        q, sc = _queue(8)
        del q  # kept: 0.94 GB
        torch.cuda.empty_cache()
        free, _ = torch.cuda.mem_get_info()
        hold = torch.empty(free - int(2.9 * GB), dtype=torch.uint8, device="cuda")
        assert engine.wq3d_queue_step(None, 1) != 0
        text = engine.wq3d_last_error_string()
        free, _ = torch.cuda.mem_get_info()
        q, sc = _queue(64)
        left, _ = torch.cuda.mem_get_info()
        assert engine.wq3d_last_error_string() == text
        # the first set was taken and nothing given back
        assert free - left > 2.0 * GB
        got = _rays(q, sc)
        for name in want:
            assert np.array_equal(got[name], want[name]), name
        assert free - torch.cuda.mem_get_info()[0] > 2.0 * GB
        del q
    finally:
        del hold
        torch.cuda.empty_cache()
        engine.wq3d_set_queue_cache(0)
        engine.wq3d_set_queue_cache(2)
