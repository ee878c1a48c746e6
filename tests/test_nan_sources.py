"""GPU: particles without a position.

With eps2 = 0, particles that coincide get accelerations that are no numbers, and
the frame after that positions: the reference sums such particles into every
force whose walk opens their leaf.  Packed and plain entries alike: frames equal
the oracle's bit for bit (where it has no number, neither does the frame).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [2, 3])
@pytest.mark.parametrize("kw", [{}, dict(min_size=1e-20), dict(temp_enabled=1),
                                dict(temp_enabled=1, min_size=1e-20)])
def test_frames_match_oracle(ge, ics, O, dims, kw):
    n = 3000
    st = ics.plummer3d(n, seed=1) if dims == 3 else ics.disk2d(n, seed=1)
    st = {k: v.copy() for k, v in st.items()}
    axes = "xyz"[:dims]
    for a in axes:
        st[a][50:53] = st[a][50]   # fewer than a leaf holds
        st["v" + a][50:53] = st["v" + a][50]
    st["temp"] = np.random.default_rng(3).uniform(100.0, 5000.0, n).astype(np.float32)
    base = dict(G=1.0, theta=0.7, eps2=0.0, dt=1e-3, leaf_cap=4)
    ref = {k: v.copy() for k, v in st.items()}
    for a in axes:
        ref["a" + a] = np.zeros(n, np.float32)
    prm = O.make_params(dims, temp_enabled=bool(kw.get("temp_enabled")),
                        **{k: v for k, v in kw.items() if k != "temp_enabled"}, **base)
    with ge.Simulation(ge.default_params(dims, precision=ge.PREC_EXACT, **kw, **base)) as s:
        s.upload({k: v for k, v in st.items() if k != "temp"})
        s.upload_temp(st["temp"])
        for _ in range(2):
            s.step(1)
            O.frame(prm, ref, walk_kind=0)
        out = s.download()
        out["temp"] = s.download_temp()
    assert np.isnan(ref["ax"]).sum() > 3
    for k in [p + a for p in ("", "v", "a") for a in axes] + ["m", "id", "temp"]:
        assert np.array_equal(out[k], ref[k], equal_nan=True), k
