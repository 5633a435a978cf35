"""Point evaluations and eigenray sums on a device whose memory is nearly all
taken: what destroyed queues left is given back to them, and one that finds
no room all the same fails alone, without an error for the next queue."""
import ctypes as C

import numpy as np
import pytest

import underseamodelinglibrary_b200 as u
from underseamodelinglibrary_b200 import _abi
from underseamodelinglibrary_b200 import scenarios as S
from underseamodelinglibrary_b200 import types as T

pytestmark = pytest.mark.gpu

N = 6_000_000
LEFT = 192 << 20  # every call below asks for more


def _calls():
    T.compute_earth_radius(45.0)
    oc = u.ocean_model(u.boundary_flat(), u.boundary_flat(800.0, u.reflect_loss_rayleigh("sand")),
                       u.profile_linear(1500.0, 0.05))
    oc.handle()
    r = T.earth_radius() - np.linspace(0.0, 800.0, N)
    z = np.full(N, 0.7)
    lib = _abi.load_engine()

    def sums():
        nt, f = N, np.array([1000.0])
        total = np.zeros(nt * C.sizeof(_abi.wq3d_eigenray), np.uint8)
        ti, tp = np.empty(nt), np.empty(nt)
        _abi.check(lib, lib.wq3d_sum_eigenrays(None, None, None, 0, _abi.as_dp(f), 1, nt, 1, 1,
                                               total.ctypes.data, _abi.as_dp(ti), _abi.as_dp(tp)))
        return ti

    return {
        "sound_speed": lambda: oc.sound_speed(r)[0],
        "height": lambda: oc.height(1, z, z)[0],
        "attenuation": lambda: oc.attenuation(r, 1000.0, np.array([1e3, 2e3, 4e3]))[:, 0],
        "reflect_loss": lambda: oc.reflect_loss(1, np.linspace(0.01, 1.5, N), np.array([1e3, 2e3]))[0][:, 0],
        "sum_eigenrays": sums,
    }


def _fill():
    import torch
    free, _ = torch.cuda.mem_get_info()
    return torch.empty(free - LEFT, dtype=torch.uint8, device="cuda")


def _small_run():
    q = S.build_queue(S.eigenray_basic(), u.wave_queue)
    q.run(1.0)
    T.compute_earth_radius(45.0)


@pytest.mark.parametrize("name", ["sound_speed", "height", "attenuation", "reflect_loss", "sum_eigenrays"])
def test_call_on_a_nearly_full_device(engine, name):
    import torch
    call = _calls()[name]
    torch.cuda.empty_cache()
    hold = None
    try:
        assert engine.wq3d_set_queue_cache(0) == 0
        _small_run()  # takes the kernels' local memory, which the device then keeps
        want = call()
        assert engine.wq3d_set_queue_cache(2) == 0
        free0, _ = torch.cuda.mem_get_info()
        sc = S.reverb_scale(100.0, 901, 91, 64, 0.2)
        qs = [S.build_queue(sc, u.wave_queue, precision=_abi.FP32C) for _ in range(2)]
        del qs
        assert free0 - torch.cuda.mem_get_info()[0] > 512 << 20  # idle, for the call to take back
        T.compute_earth_radius(45.0)  # the queues' scenario has its own
        hold = _fill()
        assert np.array_equal(call(), want)
        # nothing idle is left: the call fails, a queue that fits does not
        hold = None
        torch.cuda.empty_cache()
        assert engine.wq3d_set_queue_cache(0) == 0
        assert engine.wq3d_set_queue_cache(2) == 0
        hold = _fill()
        with pytest.raises(_abi.EngineError):
            call()
        _small_run()
    finally:
        del hold
        torch.cuda.empty_cache()
        engine.wq3d_set_queue_cache(2)
