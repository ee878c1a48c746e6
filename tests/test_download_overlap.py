"""GPU: reads of the state into page-locked arrays that share memory.

Arrays are written in the call's order, so where two of them overlap the later
one's values stand, as in pageable memory: a caller may point the arrays it does
not want at one scratch buffer.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KEYS = ("x", "y", "vx", "vy", "ax", "ay", "m", "id")


@pytest.mark.parametrize("n", [100, 9001, 200003])
@pytest.mark.parametrize("stride", [0, 0.5, 0.99, 1])
def test_later_arrays_win(ge, ics, n, stride):
    import torch
    step = int(n * stride)
    with ge.Simulation(ge.default_params(2, G=1.0, theta=0.8, eps2=1e-4, dt=1e-3)) as s:
        s.upload(ics.disk2d(n, seed=7))
        s.step(1)
        want = np.zeros(n + step * (len(KEYS) - 1), np.uint32)
        state = s.download()
        for k, name in enumerate(KEYS):
            want[step * k:step * k + n] = state[name].view(np.uint32)
        got = torch.zeros(len(want), dtype=torch.int32, pin_memory=True)
        at = {name: C.c_void_p(got.data_ptr() + 4 * step * k) for k, name in enumerate(KEYS)}
        order = ("x", "y", "z", "vx", "vy", "vz", "ax", "ay", "az", "m", "id")
        s._check(ge.lib().ge_download(s._h, *[at.get(k) for k in order]))
        assert np.array_equal(got.numpy().view(np.uint32), want)
