"""GPU: the FAST direct sum's split over warps at its edges.

Blocks of 32 particles, eight partial sums over runs of 32 sources, 512 sources
staged at a time: sizes on both sides of each, alone and batched, against the
sum in FP64.  Bound per particle: a term takes some 12 roundings, a partial sum
n / 8 additions and the last eight, so |a - a_ref| <= (20 + n / 8) 2^-24 S, S
the sum of the terms' magnitudes.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = (1, 2, 31, 32, 33, 127, 129, 255, 257, 511, 513, 1025, 4999)


def _system(ics, dims, n):
    st = ics.plummer3d(n, seed=n) if dims == 3 else ics.disk2d(max(n, 2), seed=n)
    return {k: v[:n].copy() for k, v in st.items()}


@pytest.mark.parametrize("dims", [2, 3])
@pytest.mark.parametrize("periodic", [0, 1])
def test_direct_fast_against_fp64(ge, ics, dims, periodic):
    dom = 7.0
    kw = dict(G=1.0, theta=0.7, eps2=1e-4, direct_eps2=0.02, dt=1e-3, direct_below=5000,
              precision=ge.PREC_FAST)
    if periodic:
        kw.update(periodic=1, domain=(dom, dom, dom))
    sts = [_system(ics, dims, n) for n in SIZES]
    alone = []
    for st in sts:
        with ge.Simulation(ge.default_params(dims, **kw)) as s:
            s.upload(st)
            s.step(1)
            alone.append(s.download())
    with ge.Simulation(ge.default_params(dims, **kw)) as b:
        hs = [b.add_sim(st) for st in sts]
        b.step(1)
        batch = [b.download_sim(h) for h in hs]
    names = "xyz"[:dims]
    for n, a, c in zip(SIZES, alone, batch):
        for k in a:
            assert np.array_equal(a[k], c[k]), (n, k)
        x = np.stack([a[k] for k in names])
        d = (x[:, None, :] - x[:, :, None]).astype(np.float64)   # FP32 differences: the wrap's
        if periodic:                                             # compares are on these
            d -= dom * ((d > 0.5 * dom).astype(float) - (d < -0.5 * dom).astype(float))
        f = a["m"].astype(np.float64) * ((d * d).sum(0) + np.float64(np.float32(0.02))) ** -1.5
        ref = (d * f).sum(-1)
        mag = (np.sqrt((d * d).sum(0)) * f).sum(-1)
        got = np.stack([a["a" + k] for k in names]).astype(np.float64)
        err = np.sqrt(((got - ref) ** 2).sum(0))
        assert (err <= (20 + n / 8) * 2.0 ** -24 * mag + 1e-30).all(), (n, (err / (mag + 1e-30)).max())
