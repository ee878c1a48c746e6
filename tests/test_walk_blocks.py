"""GPU: the 2D walk's block sizes.

The block size goes by the launch's particles, and a particle's walk does not
depend on it: simulations on both sides of each of its limits, alone, equal the
same simulations in one batch, whose launch takes another size, bit for bit.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KEYS = ("x", "y", "vx", "vy", "ax", "ay", "m", "id")


@pytest.mark.parametrize("exact", [False, True])
@pytest.mark.parametrize("sizes", [(1, 511, 513), (32768, 32769), (37888, 37889, 100),
                                   (151552, 151553)])
def test_alone_equals_batch(ge, ics, sizes, exact):
    prm = ge.default_params(2, G=1.0, theta=0.7, softening=0.005, dt=1e-3,
                            precision=ge.PREC_EXACT if exact else ge.PREC_FAST)
    sts = [{k: v[:n].copy() for k, v in ics.disk2d(max(n, 64), seed=80 + n % 11).items()}
           for n in sizes]
    with ge.Simulation(prm) as b:
        hs = [b.add_sim(st) for st in sts]
        b.add_sim(ics.disk2d(160000, seed=5))
        b.step(2)
        got = [b.download_sim(h) for h in hs]
    for st, g in zip(sts, got):
        with ge.Simulation(prm) as a:
            a.upload(st)
            a.step(2)
            alone = a.download()
        for k in KEYS:
            assert np.array_equal(alone[k], g[k]), k
