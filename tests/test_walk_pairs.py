"""GPU: the 3D FAST walk for two particles per thread, and the periodic walk
whose offsets cannot wrap.

Both take the same entries in the same order as the single walk with the wrap,
so everything is compared bit for bit: pairs (200,000 particles and more) with
the counting walk, which goes particle by particle, and in a batch whose
simulations meet inside a pair, one of them left to the direct sum, with each
simulation alone; the periodic walk with the oracle, on systems inside half the
domain, across it, and with negative masses (a centre of mass may then lie
outside the box).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KEYS = ("x", "y", "z", "vx", "vy", "vz", "ax", "ay", "az", "m", "id")


def _params(ge, **kw):
    base = dict(G=1.0, theta=0.8, eps2=0.01, dt=1e-3, leaf_cap=4)
    base.update(kw)
    return ge.default_params(3, **base)


@pytest.mark.parametrize("n,kw", [(200001, {}), (400001, dict(theta=1.0)),
                                  (400000, dict(periodic=1, domain=(60.0, 60.0, 60.0))),
                                  (200001, dict(min_size=1e-20))])
def test_pairs_equal_single(ge, ics, n, kw):
    st = ics.plummer3d(n, seed=51)
    st["m"][::1000] = 0.0
    outs = []
    for count in (False, True):
        with ge.Simulation(_params(ge, **kw)) as s:
            s.upload(st)
            s.count_interactions(count)
            s.step(1)
            outs.append(s.download())
    for k in KEYS:
        assert np.array_equal(outs[0][k], outs[1][k]), k


def test_pairs_in_a_batch(ge, ics):
    sizes = (120001, 4001, 100002, 1)
    sts = [{k: v[:n].copy() for k, v in ics.plummer3d(max(n, 2), seed=60 + n % 7).items()}
           for n in sizes]
    kw = dict(direct_below=5000, direct_eps2=0.01)
    with ge.Simulation(_params(ge, **kw)) as b:
        hs = [b.add_sim(st) for st in sts]
        b.step(2)
        got = [b.download_sim(h) for h in hs]
    for st, g in zip(sts, got):
        with ge.Simulation(_params(ge, **kw)) as a:
            a.upload(st)
            a.step(2)
            alone = a.download()
        for k in KEYS:
            assert np.array_equal(alone[k], g[k]), k


@pytest.mark.parametrize("dims", [2, 3])
@pytest.mark.parametrize("domain", [9.0, 16.0, 40.0])
@pytest.mark.parametrize("signs", [False, True])
def test_periodic_walk_matches_oracle(ge, ics, O, dims, domain, signs):
    st = ics.disk2d(4000, seed=71) if dims == 2 else ics.plummer3d(4000, seed=71)
    keep = np.all([np.abs(st[k]) < 4.0 for k in "xyz"[:dims]], axis=0)
    st = {k: v[keep].copy() for k, v in st.items()}
    st["id"] = np.arange(len(st["x"]), dtype=np.uint32)
    if dims == 2:
        st["x"] += np.float32(0.5 * domain)
        st["y"] += np.float32(0.5 * domain)
    if signs:
        st["m"][1::3] *= np.float32(-0.9)
    dom = (domain,) * 3
    eps2 = 1e-4 if dims == 2 else 0.01
    ref = {k: np.array(v, copy=True) for k, v in st.items()}
    for k in "xyz"[:dims]:
        ref["a" + k] = np.zeros(len(ref["x"]), np.float32)
    prm = O.make_params(dims, G=1.0, theta=0.8, eps2=eps2, dt=1e-3, leaf_cap=4, periodic=True,
                        domain=dom)
    O.frame(prm, ref, walk_kind=0)
    p = ge.default_params(dims, G=1.0, theta=0.8, eps2=eps2, dt=1e-3, leaf_cap=4, periodic=1,
                          domain=dom, precision=ge.PREC_EXACT)
    with ge.Simulation(p) as s:
        s.upload(st)
        s.step(1)
        out = s.download()
    for k in ["id"] + [a + b for a in ("", "v", "a") for b in "xyz"[:dims]]:
        assert np.array_equal(out[k], ref[k], equal_nan=True), k
