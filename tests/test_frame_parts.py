"""GPU: ge_frame_host with the walk in one, two, three and four particle ranges.

The number of ranges follows the frame's size (131,072 particles each in 2D,
200,000 in 3D, four at most); every frame equals the serial path's (upload, one
step, download) bit for bit.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,n", [(2, 131071), (2, 262145), (2, 400001), (2, 524289),
                                    (3, 399999), (3, 400001)])
def test_ranges_equal_serial(ge, ics, dims, n):
    st = ics.plummer3d(n, seed=5) if dims == 3 else ics.disk2d(n, seed=5)
    for k in "xyz"[:dims]:
        st["a" + k] = np.zeros(n, np.float32)
    ser = {k: v.copy() for k, v in st.items()}
    p = ge.default_params(dims, G=1.0, theta=1.0, softening=0.01, dt=1e-3)
    with ge.Simulation(p) as a, ge.Simulation(p) as b:
        for _ in range(2):   # the second frame is the overlapped one
            a.frame_host(st)
            b.upload(ser)
            b.step(1)
            ser = b.download()
    for k in st:
        assert np.array_equal(st[k], ser[k]), k
