"""GPU: the mixed mode's walk of groups of 32 on both sides of 200,000 particles.

Launches from there on keep six blocks per SM and load no candidates ahead; a
group's walk is the same.  A simulation alone equals itself in a batch that goes
over the limit, bit for bit, forces, counts and (to the order of its atomics) the
potential energy.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [2, 3])
@pytest.mark.parametrize("n", [1, 33, 20000, 199999])
@pytest.mark.parametrize("eps2,count", [(1e-4, False), (1e-4, True), (0.0, False)])
def test_alone_equals_batch(ge, ics, dims, n, eps2, count):
    kw = dict(G=1.0, theta=0.7, eps2=eps2, dt=1e-3, leaf_cap=8, group_size=32,
              precision=ge.PREC_MIXED)

    def sim(k, seed):
        st = ics.plummer3d(max(k, 2), seed=seed) if dims == 3 else ics.disk2d(max(k, 2), seed=seed)
        return {a: v[:k].copy() for a, v in st.items()}

    st, other = sim(n, 5), sim(200000, 6)
    with ge.Simulation(ge.default_params(dims, **kw)) as a:
        a.upload(st)
        a.count_interactions(count)
        a.step(1)
        alone, na = a.download(), a.stats().interactions
        if count and n > 1:
            ea = a.energy_f64()
    with ge.Simulation(ge.default_params(dims, **kw)) as o:
        o.upload(other)
        o.count_interactions(count)
        o.step(1)
        no = o.stats().interactions
        if count and n > 1:
            eo = o.energy_f64()
    with ge.Simulation(ge.default_params(dims, **kw)) as b:
        b.add_sim(st)
        b.add_sim(other)
        b.count_interactions(count)
        b.step(1)
        got, nb = b.download(), b.stats().interactions
        if count and n > 1:
            eb = b.energy_f64()
    for k, v in alone.items():
        assert np.array_equal(v, got[k][:n], equal_nan=True), k
    if count:
        assert na + no == nb
        if n > 1:
            assert np.allclose(np.add(ea, eo), eb, rtol=1e-12, atol=0.0), (ea, eo, eb)
