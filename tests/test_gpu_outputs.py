"""getState's device-side outputs (forces as f64 triples, kinetic energy) at sizes around the
kernels' blocks."""
import numpy as np
import pytest

import ommb200
from ommb200 import synth, systems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 85, 86, 511, 513, 40000])
def test_kinetic_energy_and_forces(n):
    rng = np.random.default_rng(n)
    mass = rng.uniform(1.0, 30.0, n)
    mass[:: max(1, n // 3)] = 0.0  # massless particles count nothing
    s = ommb200.System()
    bonds = ommb200.HarmonicBondForce()
    for i in range(n):
        s.add_particle(float(mass[i]))
    for i in range(0, n - 1, 2):
        bonds.add_bond(i, i + 1, 0.1, 1000.0)
    s.add_force(bonds)
    ctx = ommb200.Context(s, systems.langevin())
    x, v = rng.normal(size=(n, 3)), rng.normal(size=(n, 3))
    ctx.set_positions(x)
    ctx.set_velocities(v)
    st = ctx.get_state(positions=True, velocities=True, forces=True)
    # summation order only: n terms in f64
    assert abs(st.kinetic_energy - 0.5 * (mass[:, None] * v * v).sum()) <= 1e-13 * (1 + st.kinetic_energy)
    assert ctx.get_state(positions=True).kinetic_energy == st.kinetic_energy
    assert np.array_equal(st.positions, x) and np.array_equal(st.velocities, v)
    f = np.zeros((n, 3))
    i = np.arange(0, n - 1, 2)
    if len(i):
        d = x[i + 1] - x[i]
        r = np.linalg.norm(d, axis=1)
        g = (1000.0 * (r - 0.1) / r)[:, None] * d
        f[i] += g
        f[i + 1] -= g
    # one fixed-point rounding per bond end (2^-33 kJ/mol/nm) and the f64 arithmetic's
    assert np.abs(st.forces - f).max() < 1e-9


def _water(precision):
    w = synth.water_box(216, 1.9, (6, 6, 6), seed=3)
    ctx = ommb200.Context(systems.water_system(w), systems.langevin(seed=5), precision=precision)
    ctx.set_positions(w.positions)
    return ctx


def _chains(precision):
    chs = [synth.chain(n, seed=n) for n in (40, 97, 33)]
    ctx = ommb200.BatchContext([systems.chain_system(c) for c in chs],
                               systems.langevin(step_size=0.001), precision=precision)
    ctx.set_positions(np.concatenate([c.positions for c in chs]))
    return ctx


@pytest.mark.parametrize("precision", ["mixed", "double"])
@pytest.mark.parametrize("make", [_water, _chains])
def test_energy_with_and_without_the_virial(make, precision):
    ctx = make(precision)
    plain = ctx.get_state(forces=True, energy=True)
    both = ctx.get_state(forces=True, energy=True, virial=True)
    only = ctx.get_state(virial=True)
    assert plain.virial is None
    assert np.array_equal(plain.forces, both.forces)
    # the same pair energies; f64 expressions may contract differently in the two forms
    assert abs(plain.potential_energy - both.potential_energy) <= 1e-12 * abs(both.potential_energy)
    assert np.array_equal(only.virial, both.virial) and np.abs(both.virial).max() > 0.0
