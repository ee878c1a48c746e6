"""GPU: the 3D walk's block sizes.

EXACT, MIXED (per particle) and heat-exchange walks, and FAST ones over plain
entries (here from a minimum size too small for packed ones), take blocks of 1024
threads where these fill the SMs evenly, the last also from two rows on, and of
256 elsewhere.  A particle's walk does not
depend on it: simulations on both sides of the rule's limits, alone, equal the
same simulation in a batch, whose launch takes another size, bit for bit.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KEYS = ("x", "y", "z", "vx", "vy", "vz", "ax", "ay", "az", "m", "id", "temp")
ROW = 148 * 1024   # a full row of blocks


# one row: nine tenths of it are 133.2 blocks; MIXED two rows, 266.4 blocks
@pytest.mark.parametrize("mode,n", [("EXACT", 133 * 1024), ("EXACT", 133 * 1024 + 1), ("EXACT", ROW),
                                    ("EXACT", ROW + 1), ("heat", 134 * 1024), ("heat", ROW),
                                    ("EXACT heat", ROW - 3), ("EXACT periodic", ROW),
                                    ("MIXED", 266 * 1024), ("MIXED", 266 * 1024 + 1),
                                    ("plain", ROW), ("plain", 2 * ROW), ("plain", 2 * ROW + 1),
                                    ("plain", 3 * ROW // 2)])
def test_alone_equals_batch(ge, ics, mode, n):
    kw = dict(G=1.0, theta=1.0, eps2=0.01, dt=1e-3)
    if "EXACT" in mode:
        kw.update(precision=ge.PREC_EXACT)
    if "MIXED" in mode:
        kw.update(precision=ge.PREC_MIXED, group_size=0, leaf_cap=4)
    if "heat" in mode:
        kw.update(temp_enabled=1)
    if mode == "plain":
        kw.update(min_size=1e-20)
    if "periodic" in mode:
        kw.update(periodic=1, domain=(60.0,) * 3)
    st, other = ics.plummer3d(n, seed=3), ics.plummer3d(5000, seed=4)
    temp = np.random.default_rng(2).uniform(100.0, 5000.0, n + 5000).astype(np.float32)
    outs = []
    for batch in (False, True):
        with ge.Simulation(ge.default_params(3, **kw)) as s:
            if batch:
                s.add_sim(st)
                s.add_sim(other)
            else:
                s.upload(st)
            if "heat" in mode:
                s.upload_temp(temp[:n + 5000 * batch])
            s.step(2)
            out = s.download()
            if "heat" in mode:
                out["temp"] = s.download_temp()
            outs.append({k: v[:n] for k, v in out.items()})
    for k in KEYS:
        if k in outs[0]:
            assert np.array_equal(outs[0][k], outs[1][k]), k
