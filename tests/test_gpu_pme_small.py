"""PME on grids whose axes hold one larger prime factor (the direct-sum first stage of the own
transform) and in boxes of at most 4,096 particles, whose whole reciprocal part is one launch of a
thread-block cluster, against the f64 oracle (pme.rs:141-425)."""
import numpy as np
import pytest

import oracle as O
import ommb200
from ommb200 import systems

pytestmark = pytest.mark.gpu

ALPHA = 3.0


def ions(n, box, seed):
    """Alternating unit charges, jittered about a lattice, with a weak LJ core."""
    rng = np.random.default_rng(seed)
    k = int(np.ceil(n ** (1.0 / 3.0)))
    site = np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    pos = (site + 0.5 + rng.uniform(-0.2, 0.2, site.shape)) / k * box
    pos += rng.integers(-1, 2, site.shape) * box  # any lattice image is a position
    q = np.where(np.arange(n) % 2 == 0, 1.0, -1.0) * rng.uniform(0.2, 1.0, n)
    return pos, q


def system(n, q, box, grid, exceptions=()):
    s = ommb200.System()
    s.set_default_periodic_box_vectors(*np.diag(box))
    nb = ommb200.NonbondedForce()
    nb.set_nonbonded_method("PME")
    nb.set_cutoff_distance(0.8)
    nb.set_pme_parameters(ALPHA, *grid)
    nb.set_use_dispersion_correction(False)
    nb.set_reciprocal_space_force_group(1)
    for i in range(n):
        s.add_particle(20.0)
        nb.add_particle(float(q[i]), 0.2, 0.1)
    s.add_force(nb)
    return s


def check(n, box, grid, precision, scale=1.0, **options):
    box = np.asarray(box)
    pos, q = ions(n, box, seed=n + grid[0])
    q = scale * q
    ctx = ommb200.Context(system(n, q, box, grid), systems.langevin(seed=3), precision=precision,
                          **options)
    ctx.set_positions(pos)
    st = ctx.get_state(forces=True, energy=True, groups=1 << 1)
    f_ref, e_ref = O.nonbonded(pos, q, np.full(n, 0.2), np.zeros(n), method="PME", cutoff=0.8,
                               box=np.diag(box), pme=(ALPHA, grid), include_direct=False,
                               use_dispersion_correction=False)
    err = np.sqrt(((st.forces - f_ref) ** 2).sum() / (f_ref ** 2).sum())
    bound = 5e-6 if precision == "mixed" else 1e-9
    assert err < bound
    assert abs(st.potential_energy - e_ref) < bound * max(abs(e_ref), 1.0)
    ctx.close()
    return st


@pytest.mark.parametrize("precision", ["mixed", "double"])
@pytest.mark.parametrize("grid", [(11, 13, 17), (22, 26, 33), (19, 23, 29), (31, 24, 39), (62, 58, 46),
                                  (37, 22, 25)])
@pytest.mark.parametrize("bricks", [-1, 0])
def test_prime_grids(grid, precision, bricks):
    # bricks = 0 asks for the launch chain, -1 lets the cluster form take it; 37 is past the
    # largest prime of the own transform
    check(350, (1.7, 2.1, 1.9), grid, precision, pme_bricks=bricks)


@pytest.mark.parametrize("precision", ["mixed", "double"])
@pytest.mark.parametrize("n,grid", [(1, (5, 5, 5)), (2, (6, 5, 7)), (511, (16, 16, 16)),
                                    (513, (17, 15, 40)), (1500, (23, 23, 23)),
                                    (4095, (33, 34, 35)), (4096, (40, 30, 36)),
                                    (4097, (33, 34, 35))])
def test_cluster_sizes(n, grid, precision):
    # the last two particle counts are past the cluster form's; 17 planes over 16 CTAs leave some
    # CTAs without planes
    check(n, (2.6, 2.4, 2.5), grid, precision)


@pytest.mark.parametrize("precision", ["mixed", "double"])
@pytest.mark.parametrize("scale", [2.5, 30.0])
@pytest.mark.parametrize("bricks", [-1, 0])
def test_charges_on_both_sides_of_the_staged_limits(precision, scale, bricks):
    # |q| from 0.5 to 2.5 e and from 6 to 30 e: the staged spread takes those below 2 e (FP32) or
    # 16 e (FP64), the others go to the grid one by one
    check(300, (1.9, 1.9, 1.9), (20, 21, 22), precision, scale=scale, pme_bricks=bricks)


def test_charges_beyond_the_shared_sums_take_the_launch_chain():
    # sum |q| above the cluster form's limit, reached through a parameter update; back below it
    # the forces are the first ones again
    n, box, grid = 300, np.array([1.8, 1.9, 2.0]), (18, 20, 22)
    pos, q = ions(n, box, 5)
    ctx = ommb200.Context(system(n, q, box, grid), systems.langevin(seed=3))
    ctx.set_positions(pos)
    before = ctx.get_state(forces=True, groups=1 << 1).forces

    def update(charges):
        nb = ommb200.NonbondedForce()
        for c in charges:
            nb.add_particle(float(c), 0.2, 0.1)
        ctx.update_nonbonded_parameters(nb)

    big = q * (9000.0 / np.abs(q).sum())
    update(big)
    st = ctx.get_state(forces=True, energy=True, groups=1 << 1)
    f_ref, _ = O.nonbonded(pos, big, np.full(n, 0.2), np.zeros(n), method="PME", cutoff=0.8,
                           box=np.diag(box), pme=(ALPHA, grid), include_direct=False,
                           use_dispersion_correction=False)
    assert np.sqrt(((st.forces - f_ref) ** 2).sum() / (f_ref ** 2).sum()) < 5e-6
    update(q)
    assert np.array_equal(ctx.get_state(forces=True, groups=1 << 1).forces, before)


def test_cluster_trajectory_equals_the_launch_chain():
    # the same fixed-point grid, transform and per-particle sums up to FP32 rounding
    n, box, grid = 1000, np.array([2.4, 2.4, 2.4]), (22, 23, 24)
    pos, q = ions(n, box, 9)
    out = []
    for bricks in (-1, 0):
        ctx = ommb200.Context(system(n, 0.3 * q, box, grid), systems.langevin(seed=3, step_size=0.001),
                              pme_bricks=bricks)
        ctx.set_positions(pos)
        ctx.set_velocities_to_temperature(300.0, seed=2)
        ctx.step(60)  # rebuilds beside the reciprocal part, from a graph
        out.append(ctx.get_state(positions=True).positions)
        ctx.close()
    assert np.abs(out[0] - out[1]).max() < 1e-5
