"""GPU: contexts whose walks read different layouts of the same tree.

3D builds pack their entries' sizes and successors into one word, except where
the walk is faster without (heat exchange, the warp walk).  Frames that go back
and forth between the two in one context equal the oracle's bit for bit, or those
of a context for each.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KEYS = ("x", "y", "z", "vx", "vy", "vz", "ax", "ay", "az", "m", "id", "temp")


@pytest.mark.parametrize("n", [1, 2, 33, 4099])
@pytest.mark.parametrize("periodic", [False, True])
def test_heat_on_and_off(ge, ics, O, n, periodic):
    st = {k: v[:n].copy() for k, v in ics.plummer3d(max(n, 2), seed=n).items()}
    st["temp"] = np.random.default_rng(n).uniform(100.0, 5000.0, n).astype(np.float32)
    kw = dict(G=1.0, theta=0.7, eps2=0.01, dt=1e-3, leaf_cap=4)
    dom = dict(domain=(60.0,) * 3)
    ref = {k: v.copy() for k, v in st.items()}
    for k in "xyz":
        ref["a" + k] = np.zeros(n, np.float32)
    with ge.Simulation(ge.default_params(3, precision=ge.PREC_EXACT, temp_enabled=1,
                                         periodic=int(periodic), **dom, **kw)) as s:
        s.upload({k: v for k, v in st.items() if k != "temp"})
        s.upload_temp(st["temp"])
        for heat in (True, False, True, True, False):
            s.set_params(ge.default_params(3, precision=ge.PREC_EXACT, temp_enabled=int(heat),
                                           heat_cond=0.045, periodic=int(periodic), **dom, **kw))
            s.step(1)
            O.frame(O.make_params(3, temp_enabled=heat, heat_cond=0.045, periodic=periodic,
                                  **dom, **kw), ref, walk_kind=0)
            out = s.download()
            out["temp"] = s.download_temp()
            for k in KEYS:
                assert np.array_equal(out[k], ref[k]), (heat, k)


@pytest.mark.parametrize("n", [1, 2, 33, 4099, 30001])
def test_warp_walk_on_and_off(ge, ics, n):
    """Forces on one state by either walk, switched before the build: each as
    from a context that only knows that walk."""
    st = {k: v[:n].copy() for k, v in ics.plummer3d(max(n, 2), seed=n).items()}

    def params(kind):
        return ge.default_params(3, G=1.0, theta=0.6, eps2=0.01, dt=1e-3, walk_kind=kind)

    def forces(s):
        s.compute_morton_keys()
        s.sort_particles_by_morton_key()
        s.build_tree()
        s.calculate_force_from_grid()
        return s.download()

    alone = []
    for kind in (0, 1):
        with ge.Simulation(params(kind)) as s:
            s.upload(st)
            alone.append(forces(s))
    with ge.Simulation(params(0)) as s:
        s.upload(st)
        for kind in (1, 0, 1, 1, 0):
            s.set_params(params(kind))
            out = forces(s)
            for k in KEYS[:-1]:
                assert np.array_equal(out[k], alone[kind][k]), (kind, k)
