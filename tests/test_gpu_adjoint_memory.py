"""A reverse sweep whose workspace finds no room fails with an error, and the
same call gives the gradient once there is room again: a workspace is made
whole or not at all.  (Half a workspace would leave null addresses that the
next call took for buffers.)"""
import numpy as np
import pytest

from underseamodelinglibrary_b200 import _abi
from underseamodelinglibrary_b200 import adjoint as A

pytestmark = pytest.mark.gpu


def test_sweep_after_one_that_found_no_memory(engine):
    import torch
    # 81,991 rays, segments of 400 steps: 4.7 GB of states, then 5.5 GB of seeds
    sc = A.AdjointScenario(num_de=901, num_az=91, n_steps=60, n_targets=12, max_range=3e3)
    p = A.Propagation(sc, A.munk_nodes(), checkpoint=400)
    q = A.Propagation(sc, A.munk_nodes(), checkpoint=400)
    assert len(p.eigenrays) > 0
    w = np.ones(len(p.eigenrays))
    want = p.vjp(w, w)[0]
    del p
    assert engine.wq3d_set_queue_cache(0) == 0
    hold = None
    try:
        free, _ = torch.cuda.mem_get_info()
        hold = torch.empty(int(free - 7 * 2 ** 30), dtype=torch.uint8, device="cuda")
        for _ in range(2):
            with pytest.raises(_abi.EngineError):
                q.vjp(w, w)
        hold = None
        torch.cuda.empty_cache()
        got = q.vjp(w, w)[0]
        assert np.abs(want).max() > 0
        assert np.abs(got - want).max() <= 1e-9 * np.abs(want).max()
    finally:
        del hold
        torch.cuda.empty_cache()
        engine.wq3d_set_queue_cache(2)
