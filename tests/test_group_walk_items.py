"""GPU: the group walk's packed passes and work items at their edges.

With interaction counting off, groups of 64 and 128 are walked in items of 64
particles whose lanes take two particles in packed arithmetic, or one when the
item holds at most 32.  Sizes around the 32-particle chunks (a small system is
one group: its root), leaf capacities whose opened leaves cross the staged
list's 64 entries, and a leaf larger than a group (coincident particles down
to the minimum cell), against the oracle's group walk in FP64.

The bound is a forward error bound per particle: a term takes some 30 FP32
operations and a list pass adds up to 64 of them in turn (the passes' sums are
compensated), so |a - a_ref| <= (30 + 64 + a margin of 34) 2^-24 S with S the
sum of the terms' magnitudes, taken as the direct sum of m |d| / r^3: it holds
where the terms cancel too (a disk's central mass), and a source left out or
taken twice stands far above it.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(ge, O, st, dims, theta, eps2, gs, leaf):
    p = ge.default_params(dims, G=1.0, theta=theta, eps2=eps2, leaf_cap=leaf, dt=1e-3,
                          precision=ge.PREC_MIXED, group_size=gs)
    with ge.Simulation(p) as s:
        s.upload(st)
        s.compute_morton_keys()
        s.sort_particles_by_morton_key()
        s.build_tree()
        s.calculate_force_from_grid()
        out = s.download()
    z = out.get("z")
    bb = O.bbox(out["x"], out["y"], z)
    tree = O.build_tree(out["x"], out["y"], out["m"], bb, z=z, leaf_cap=leaf, holder=True)
    op = O.make_params(dims, G=1.0, theta=theta, eps2=eps2, leaf_cap=leaf)
    ref = O.walk_group(out["x"], out["y"], out["m"], tree, op, group_size=gs, z=z)
    got = np.stack([out["a" + k] for k in "xyz"[:dims]]).astype(np.float64)
    err = np.sqrt(((got - np.stack(ref[:dims])) ** 2).sum(0))
    x = np.stack([out[k] for k in "xyz"[:dims]]).astype(np.float64)
    d2 = sum((x[k][:, None] - x[k][None, :]) ** 2 for k in range(dims))
    size = (out["m"].astype(np.float64) * np.sqrt(d2) * (d2 + eps2) ** -1.5).sum(1)
    worst = float((err / size).max() * 2.0 ** 24)
    print(f"largest error: {worst:.1f} of 128 roundings of the terms' magnitudes")
    assert worst <= 128.0


@pytest.mark.parametrize("dims", [2, 3])
@pytest.mark.parametrize("n,gs,leaf", [(2, 64, 1), (31, 64, 4), (33, 64, 16), (65, 64, 32),
                                       (64, 128, 1), (97, 128, 16), (129, 128, 8),
                                       (9001, 64, 32), (9001, 128, 16)])
def test_items_match_oracle(ge, ics, O, dims, n, gs, leaf):
    st = ics.disk2d(n, seed=6) if dims == 2 else ics.plummer3d(n, seed=6)
    _check(ge, O, st, dims, 0.6, 1e-4 if dims == 2 else 0.01, gs, leaf)


@pytest.mark.parametrize("dims,gs", [(2, 64), (3, 128)])
def test_leaf_larger_than_a_group(ge, ics, O, dims, gs):
    """200 coincident particles beside a galaxy: one leaf of minimum size, cut
    into group-size pieces, and staged in several lists by whoever opens it."""
    st = ics.disk2d(3000, seed=7) if dims == 2 else ics.plummer3d(3000, seed=7)
    for k in "xyz"[:dims]:
        st[k][100:300] = np.float32(0.37)
    _check(ge, O, st, dims, 0.6, 1e-3 if dims == 2 else 0.01, gs, 16)
