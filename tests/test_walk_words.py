"""GPU: packed walk words against the plain layout, FAST and EXACT, 2D and 3D.

min_size = 1e-20 forces the plain layout without changing these trees, so every
output has to be equal bit for bit: in an ordinary system (in 2D the loop that
decides every entry by one signed compare), with massless particles and whole
massless nodes (the marker levels), with a root so large beside eps2 that the
markers need their own test, with theta = 0 (nothing but particles accepted),
in a periodic domain, and with a pin and a batch of two root sizes.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(ge, dims, sts, min_size, mode, kw, steps=2):
    p = ge.default_params(dims, G=1.0, dt=1e-3, leaf_cap=4, min_size=min_size,
                          precision=getattr(ge, "PREC_" + mode), **kw)
    with ge.Simulation(p) as s:
        for st in sts:
            s.add_sim(st)
        s.step(steps)
        out = s.download()
        if len(sts) == 1 and not kw.get("periodic"):
            pos = np.stack([sts[0][k][:4] for k in "xyz"[:dims]], 1) + np.float32(0.25)
            out["path"] = s.predict_trajectory(pos, np.zeros_like(pos), np.ones(4, np.float32),
                                               20, 1e-3)
    return out


@pytest.mark.parametrize("mode", ["FAST", "EXACT"])
@pytest.mark.parametrize("dims", [2, 3])
@pytest.mark.parametrize("case", ["plain", "massless", "large_root", "theta0", "periodic", "batch"])
def test_packed_equals_plain(ge, ics, dims, case, mode):
    n = 700 if case == "theta0" else 6000
    st = ics.plummer3d(n, seed=21) if dims == 3 else ics.disk2d(n, seed=21)
    kw = dict(theta=0.7, eps2=1e-4 if dims == 2 else 0.01)
    sts = [st]
    if case == "massless":
        st["m"][::3] = 0.0
        st["m"][st["x"] > 0.5] = 0.0
    elif case == "large_root":   # root 1e17: marker size^2 = 1e34 2^-124 > theta^2 eps2
        for k in "xyz"[:dims]:
            st[k][5:9] = np.float32(5e16) * np.array([-1, -1, 1, 1], np.float32)
        kw["eps2"] = 1e-12
    elif case == "theta0":
        kw["theta"] = 0.0
    elif case == "periodic":
        kw.update(periodic=1, domain=(40.0, 40.0, 40.0))
        if dims == 2:
            st["x"] += np.float32(20.0)
            st["y"] += np.float32(38.0)   # straddles the domain's edge
    elif case == "batch":
        big = ics.plummer3d(900, seed=22) if dims == 3 else ics.disk2d(900, seed=22)
        for k in "xyz"[:dims]:
            big[k] = (big[k] * np.float32(1e6)).astype(np.float32)
        sts.append(big)
    # (EXACT divides by the particle's own mass, as the reference does: after one
    # step the massless ones are NaN, share one key and the tree goes down to
    # min_size there)
    steps = 1 if case == "massless" else 2
    packed = _run(ge, dims, sts, 1e-6, mode, kw, steps)
    plain = _run(ge, dims, sts, 1e-20, mode, kw, steps)
    for k in packed:
        assert np.array_equal(packed[k], plain[k], equal_nan=True), k
