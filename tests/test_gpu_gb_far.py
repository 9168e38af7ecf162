"""The FP32 GB descreening passes at the sizes where their forms meet: partly filled blocks, one
and two blocks, and pairs on both sides of the distance from which the descreening integral and
its gradient come from their power series (|s| <= r / 4 and rho <= 3 r / 4), overlapping and
engulfed spheres among them; without a cutoff, and with one whose tiles are mostly too far apart
to hold a pair.  Against the f64 oracle (gbsa_obc.rs:184-309) with the mixed form's bound."""
import numpy as np
import pytest

import oracle as O
import ommb200
from ommb200 import synth, systems
from test_gpu_gbsa import gb_context, rms_rel

pytestmark = pytest.mark.gpu


def particles(n, spread, seed):
    rng = np.random.default_rng(seed)
    pos = np.zeros((n, 3))
    k = 0
    while k < n:  # no two closer than 0.08 nm
        p = rng.uniform(0.0, spread, 3)
        if k == 0 or ((pos[:k] - p) ** 2).sum(1).min() > 0.08 ** 2:
            pos[k] = p
            k += 1
    q = rng.normal(0.0, 0.4, n)
    radius = rng.uniform(0.1, 0.3, n)
    scale = rng.uniform(0.5, 1.2, n)
    radius[:: max(1, n // 5)] = 0.011  # a scaled radius near zero
    return pos, q, radius, scale


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 65, 200])
@pytest.mark.parametrize("spread", [1.2, 6.0])
@pytest.mark.parametrize("method", [0, 1, 2])
def test_descreening_forms_match_the_oracle(n, spread, method):
    pos, q, r, s = particles(n, spread, seed=n)
    box = np.diag([max(spread, 2.2)] * 3) if method == 2 else None
    f_ref, e_ref, _ = O.gbsa_obc(pos, q, r, s, method=method, cutoff=1.0, box=box)
    ctx = gb_context(pos, q, r, s, method=method, cutoff=1.0, box=box, precision="mixed")
    st = ctx.get_state(forces=True, energy=True)
    if np.abs(f_ref).max() > 0.0:  # no pair within the cutoff: no force at all
        assert rms_rel(st.forces, f_ref) < 5e-6
    else:
        assert np.all(st.forces == 0.0)
    assert abs(st.potential_energy - e_ref) < 5e-6 * max(1.0, abs(e_ref))


@pytest.mark.parametrize("atoms", [97, 640, 1500])
@pytest.mark.parametrize("precision,bound", [("double", 1e-9), ("mixed", 5e-6)])
def test_cutoff_chain_skips_only_empty_tiles(atoms, precision, bound):
    ch = synth.chain(atoms, seed=atoms)
    n, cutoff = ch.n_atoms, 0.9
    ctx = ommb200.Context(systems.chain_system(ch, cutoff=cutoff), systems.langevin(),
                          precision=precision)
    # far from the origin, where FP32 coordinates round most
    pos = ch.positions + np.array([40.0, -25.0, 60.0])
    ctx.set_positions(pos)
    st = ctx.get_state(forces=True, energy=True)
    if precision == "mixed":  # the oracle sees the positions as the FP32 kernels round them
        pos = pos.astype(np.float32).astype(np.float64)
    excl = sorted({(i, i + 1) for i in range(n - 1)} | {(i, i + 2) for i in range(n - 2)})
    exc = [(i, j, 0.0, ch.sigma, 0.0) for i, j in excl]
    exc += [(i, i + 3, ch.charges[i] * ch.charges[i + 3], ch.sigma, ch.epsilon) for i in range(n - 3)]
    f1, e1 = O.nonbonded(pos, ch.charges, [ch.sigma] * n, [ch.epsilon] * n, exc,
                         method="CutoffNonPeriodic", cutoff=cutoff)
    f4, e4, _ = O.gbsa_obc(pos, ch.charges, ch.radii, [ch.gb_scale] * n, method=1, cutoff=cutoff,
                           solvent_dielectric=78.5, solute_dielectric=1.0)
    true = ch.positions + np.array([40.0, -25.0, 60.0])
    f2, e2 = O.harmonic_bonds(true, ch.bonds())
    f3, e3 = O.harmonic_angles(true, ch.angles())
    if precision == "double":
        assert rms_rel(st.forces, f1 + f2 + f3 + f4) < bound
        assert abs(st.potential_energy - (e1 + e2 + e3 + e4)) < 1e-9 * abs(e1 + e2 + e3 + e4) + 1e-6
    else:
        # the pairs a wrongly skipped tile would lose weigh thousands of times this; positions
        # near 60 nm carry 4e-6 nm of rounding, 1e-5 of a bond, in the 1-4 terms and near pairs
        total = f1 + f2 + f3 + f4
        assert rms_rel(st.forces, total) < 2e-4
