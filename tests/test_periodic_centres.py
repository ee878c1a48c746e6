"""GPU: the periodic walk where a centre of mass lies outside its root box.

The walk leaves out the wrap for a particle that no offset of anything inside
the box can carry past half the domain.  A centre of mass is a quotient of two
plain FP32 sums, and the sums of one leaf with many particles drift apart: here
a mass of 2^24 followed by ones stays at 2^24 while the first moment grows by 1
for each 0.9 (by 0.5 for each 0.45), which puts the centre up to 5 % of the domain
past the corner: past half the domain from a particle that is 0.46 from it.
The frame equals the oracle's bit for bit all the same.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# (dims, particles, where all but the last are, where the last is)
@pytest.mark.parametrize("dims,n,at,last", [(2, 800000, 0.9, 0.445), (3, 1200000, -0.45, 0.02),
                                            (2, 1000, 0.9, 0.445), (3, 1000, -0.45, 0.02)])
def test_centre_outside_the_box(ge, O, dims, n, at, last):
    st = {}
    for k in "xyz"[:dims]:
        st[k] = np.full(n, at, np.float32)
        st[k][-1] = last
        st["v" + k] = np.zeros(n, np.float32)
    st["m"] = np.ones(n, np.float32)
    st["m"][0] = 2.0 ** 24
    st["id"] = np.arange(n, dtype=np.uint32)
    kw = dict(G=1e-6, theta=0.8, eps2=4.0, dt=1e-3, leaf_cap=4)
    ref = {k: v.copy() for k, v in st.items()}
    for k in "xyz"[:dims]:
        ref["a" + k] = np.zeros(n, np.float32)
    O.frame(O.make_params(dims, periodic=True, domain=(1.0,) * 3, **kw), ref, walk_kind=0)
    p = ge.default_params(dims, periodic=1, domain=(1.0,) * 3, precision=ge.PREC_EXACT, **kw)
    with ge.Simulation(p) as s:
        s.upload(st)
        s.step(1)
        out = s.download()
    for k in ["id"] + [a + b for a in ("", "v", "a") for b in "xyz"[:dims]]:
        assert np.array_equal(out[k], ref[k]), k
