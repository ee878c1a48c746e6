"""GPU: the one-launch front (kick, box, keys, sort, gather) of small simulations.

Frames of up to 32,768 particles go through one thread-block cluster per
simulation (ge_front.cu); larger ones, and batches of too many blocks, through
one kernel per pass.  The sizes stand at the edges of the clusters (1 .. 16
blocks of 512 threads, 1, 2 or 4 particles per thread) and on both sides of
the limit; everything is compared bit for bit with the oracle's frames, or,
where the oracle has no such frame (a batch), with each simulation alone in a
context whose own route differs.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _keys(dims):
    return ["x", "y", "vx", "vy", "ax", "ay", "m", "id"] + (["z", "vz", "az"] if dims == 3 else [])


@pytest.mark.parametrize("dims,n", [(2, 1), (2, 2), (2, 33), (2, 512), (2, 513), (2, 1025),
                                    (2, 8192), (2, 8193), (2, 16385), (2, 32767), (2, 32768),
                                    (2, 32769), (3, 1), (3, 511), (3, 1024), (3, 4097),
                                    (3, 8193), (3, 16385)])
def test_frames_match_oracle(ge, ics, O, dims, n):
    st = ics.plummer3d(n, seed=n) if dims == 3 else ics.disk2d(max(n, 2), seed=n)
    st = {k: v[:n].copy() for k, v in st.items()}
    if n >= 513:   # a run of coincident particles: equal keys keep their order
        for k in "xyz"[:dims]:
            st[k][100:400] = st[k][100]
            st["v" + k][100:400] = st["v" + k][100]
    steps = 3 if n <= 8193 else 1
    eps2 = 1e-4 if dims == 2 else 0.01
    ref = {k: np.array(v, copy=True) for k, v in st.items()}
    for k in "xyz"[:dims]:
        ref["a" + k] = np.zeros(n, np.float32)
    prm = O.make_params(dims, G=1.0, theta=0.8, eps2=eps2, dt=1e-3, leaf_cap=4)
    for _ in range(steps):
        O.frame(prm, ref, walk_kind=0)
    p = ge.default_params(dims, G=1.0, theta=0.8, eps2=eps2, dt=1e-3, leaf_cap=4,
                          precision=ge.PREC_EXACT)
    with ge.Simulation(p) as s:
        s.upload(st)
        s.step(steps)
        out = s.download()
    for k in _keys(dims):
        assert np.array_equal(out[k], ref[k]), k


@pytest.mark.parametrize("dims,sizes", [(2, (1, 700, 5000, 32768)), (3, (2, 513, 9000)),
                                        (2, (40000, 3, 600))])
@pytest.mark.parametrize("mode", ["FAST", "MIXED"])
def test_batch_equals_alone(ge, ics, dims, sizes, mode):
    """Simulations of one batch (one launch, or per pass where one of them is
    too large) against each alone; pins, previous velocities and compensation
    terms travel along."""
    kw = dict(G=1.0, theta=0.8, eps2=1e-4, dt=1e-3, leaf_cap=4, track_prev_vel=1,
              precision=getattr(ge, "PREC_" + mode))
    def sim(n, k):
        st = ics.plummer3d(n, seed=k) if dims == 3 else ics.disk2d(max(n, 2), seed=k)
        return {a: v[:n].copy() for a, v in st.items()}
    sts = [sim(n, 40 + k) for k, n in enumerate(sizes)]
    pin = [(np.arange(n) % 7 == 3).astype(np.uint8) for n in sizes]
    with ge.Simulation(ge.default_params(dims, **kw)) as b:
        for st in sts:
            b.add_sim(st)
        b.upload_pinned(np.concatenate(pin))
        b.step(5)
        whole = b.download_state()
    at = 0
    for st, pn, n in zip(sts, pin, sizes):
        with ge.Simulation(ge.default_params(dims, **kw)) as a:
            a.upload(st)
            a.upload_pinned(pn)
            a.step(5)
            alone = a.download_state()
        for k, v in alone.items():
            assert np.array_equal(v, whole[k][at:at + n]), (n, k)
        at += n
