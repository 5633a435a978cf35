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
