"""The three-launch neighbour-list rebuild: columns that are empty, partly filled and full, boxes
too small for the nearest image alone, elongated boxes (few columns, long sorts), clumps that
overflow and grow, and a triclinic box turned rectangular and back; the interacting pairs must be
the reference's (neighbors.rs:96-181) and the forces the oracle's."""
import numpy as np
import pytest

import oracle as O
import ommb200
from ommb200 import systems

pytestmark = pytest.mark.gpu

RC = 0.6


def context(n, box, seed=5, **kw):
    s = ommb200.System()
    s.set_default_periodic_box_vectors(*np.asarray(box))
    nb = ommb200.NonbondedForce()
    nb.set_nonbonded_method("CutoffPeriodic")
    nb.set_cutoff_distance(RC)
    nb.set_use_dispersion_correction(False)
    for i in range(n):
        s.add_particle(12.0)
        nb.add_particle(0.2 * (-1) ** i, 0.2, 0.3)
    for i in range(0, n - 1, 5):
        nb.add_exception(i, i + 1, 0.0, 0.2, 0.0)
    s.add_force(nb)
    return ommb200.Context(s, systems.langevin(seed=seed, step_size=0.001), **kw)


def spread(n, box, seed, lo=0.0, hi=1.0):
    """n points in the [lo, hi) part of each axis, no two closer than about 0.15 nm."""
    rng = np.random.default_rng(seed)
    length = np.diag(np.asarray(box)) * (hi - lo)
    k = np.maximum(1, np.floor(length / 0.17)).astype(int)
    sites = rng.permutation(int(k.prod()))[:n]
    assert len(sites) == n
    ijk = np.stack([sites // (k[1] * k[2]), (sites // k[2]) % k[1], sites % k[2]], 1)
    pos = (ijk + 0.5 + rng.uniform(-0.05, 0.05, (n, 3))) * length / k + lo * np.diag(np.asarray(box))
    return pos + rng.integers(-2, 3, (n, 3)) @ np.asarray(box, float)  # any image


def check(ctx, pos, box):
    n = len(pos)
    ctx.set_positions(pos)
    exc = [(i, i + 1, 0.0, 0.2, 0.0) for i in range(0, n - 1, 5)]
    f_ref, e_ref = O.nonbonded(pos, [0.2 * (-1) ** i for i in range(n)], [0.2] * n, [0.3] * n, exc,
                               method="CutoffPeriodic", cutoff=RC, box=np.asarray(box),
                               use_dispersion_correction=False)
    st = ctx.get_state(forces=True, energy=True)
    if np.abs(f_ref).max() > 0:
        assert np.sqrt(((st.forces - f_ref) ** 2).sum() / (f_ref ** 2).sum()) < 5e-6
    # the total nearly cancels: a particle's 50 to 100 pair energies of up to some tens of kJ/mol
    # round in FP32 (6e-8) with their distances (a few 1e-7), 2e-5 kJ/mol a particle if all add up
    assert abs(st.potential_energy - e_ref) < 1e-5 * abs(e_ref) + 2e-5 * n + 1e-5
    want = O.pair_set(pos, RC, np.asarray(box), [(i, i + 1) for i in range(0, n - 1, 5)])
    got = ctx.debug_pair_list()
    key = lambda p: np.sort(np.sort(np.asarray(p), 1) @ np.array([n, 1]))  # noqa: E731
    assert np.array_equal(key(got) if len(got) else np.zeros(0), key(want) if len(want) else np.zeros(0))


@pytest.mark.parametrize("precision", ["mixed", "double"])
@pytest.mark.parametrize("n,box", [(1, (1.3, 1.3, 1.3)), (33, (1.25, 1.3, 1.4)), (257, (1.3, 1.9, 1.25)),
                                   (1000, (2.0, 2.4, 2.9)), (700, (1.3, 1.3, 9.0)),
                                   (900, (9.0, 1.4, 1.3)), (40, (6.0, 6.0, 6.0))])
def test_sizes_and_shapes(n, box, precision):
    box = np.diag(box)
    ctx = context(n, box, precision=precision)
    check(ctx, spread(n, box, seed=n), box)
    # the whole system in one corner: full columns beside empty ones, the list may have to grow
    if n <= 40 or n == 1000:
        part = 0.8 if n == 1000 else 0.9
        check(ctx, spread(n, box, seed=n + 1, hi=part), box)
    check(ctx, spread(n, box, seed=n + 2), box)
    ctx.step(25)
    st = ctx.get_state(positions=True)
    check(ctx, st.positions, box)


def test_triclinic_box_turned_rectangular_and_back():
    tri = np.array([[2.4, 0, 0], [0.2, 2.3, 0], [-0.1, 0.15, 2.5]])
    rect = np.diag([2.4, 2.3, 2.5])
    n = 600
    ctx = context(n, tri)
    for k, box in enumerate((tri, rect, tri, rect)):
        ctx.set_periodic_box_vectors(*box)
        check(ctx, spread(n, box, seed=20 + k), box)
