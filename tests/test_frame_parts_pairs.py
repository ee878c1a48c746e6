"""GPU: ge_frame_host on 3D frames whose walk takes two particles per thread.

From 400,000 particles on a 3D frame's walk goes in ranges of 200,000 and more,
each a launch of its own that starts in the middle of the system; at ordinary
opening angles each range takes two particles per thread, the last one with an
odd number of them.  Every frame equals the serial path's (upload, one step,
download) bit for bit.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,theta", [(400000, 0.7), (401001, 0.7), (602001, 0.8)])
def test_ranges_equal_serial(ge, ics, n, theta):
    st = ics.plummer3d(n, seed=5)
    for k in "xyz":
        st["a" + k] = np.zeros(n, np.float32)
    ser = {k: v.copy() for k, v in st.items()}
    p = ge.default_params(3, G=1.0, theta=theta, softening=0.01, dt=1e-3)
    with ge.Simulation(p) as a, ge.Simulation(p) as b:
        for _ in range(2):   # the second frame is the overlapped one
            a.frame_host(st)
            b.upload(ser)
            b.step(1)
            ser = b.download()
    for k in st:
        assert np.array_equal(st[k], ser[k]), k
