"""GPU: reads of the state into page-locked arrays.

Up to 262,144 particles a read into page-locked arrays is one kernel's stores;
everything else (pageable memory, arrays that no single page-locked allocation
holds, odd addresses, larger states) is a copy per array.  Every form gives the
pageable read's bytes and touches nothing beside its arrays.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KEYS = ("x", "y", "vx", "vy", "ax", "ay", "m", "id")


def _args(out, dims3=False):
    order = ("x", "y", "z", "vx", "vy", "vz", "ax", "ay", "az", "m", "id")
    return [C.c_void_p(out[k].ctypes.data) if k in out else None for k in order]


def _read(ge, s, n, locked, shift):
    """One buffer of guarded arrays per key, `shift` bytes off its alignment."""
    import torch
    out, raw, keep = {}, {}, []
    for k in KEYS:
        size = 4 * n + 64
        t = torch.full((size,), 0xA5, dtype=torch.uint8, pin_memory=locked)
        keep.append(t)
        raw[k] = t.numpy()
        out[k] = raw[k][16 + shift:16 + shift + 4 * n]
    s._check(ge.lib().ge_download(s._h, *_args(out)))
    for k in KEYS:
        assert (raw[k][:16 + shift] == 0xA5).all() and (raw[k][16 + shift + 4 * n:] == 0xA5).all()
    return {k: v.tobytes() for k, v in out.items()}


@pytest.mark.parametrize("n", [1, 33, 4097, 262144, 262145])
def test_locked_reads_equal_pageable(ge, ics, n):
    st = {k: v[:n].copy() for k, v in ics.disk2d(max(n, 2), seed=31).items()}
    with ge.Simulation(ge.default_params(2, G=1.0, theta=0.8, eps2=1e-4, dt=1e-3)) as s:
        s.upload(st)
        s.step(1)
        want = {k: s.download()[k].tobytes() for k in KEYS}
        for locked in (True, False):
            for shift in (0, 4, 2):
                assert _read(ge, s, n, locked, shift) == want, (locked, shift)
        mixed = {k: v for k, v in s.download().items()}   # one array page-locked, the others not
        import torch
        t = torch.zeros(n, dtype=torch.float32, pin_memory=True)
        mixed["vx"] = t.numpy()
        s._check(ge.lib().ge_download(s._h, *_args(mixed)))
        assert {k: mixed[k].tobytes() for k in KEYS} == want

