"""The two FP32 forms of the tile pair kernel: four i-particles per lane for periodic lists, two for
the whole-block tiles of non-periodic systems.  In a box so large that no image counts both must
give the reference's pairs (neighbors.rs:96-181) and the oracle's forces, at the edges of a block."""
import numpy as np
import pytest

import oracle as O
import ommb200
from ommb200 import systems

pytestmark = pytest.mark.gpu

RC = 0.9
BOXES = {"rectangular": np.diag([6.0, 6.5, 7.0]),
         "triclinic": np.array([[6.0, 0, 0], [0.5, 6.5, 0], [-0.4, 0.6, 7.0]])}


@pytest.mark.parametrize("n", [1, 2, 16, 17, 31, 32, 33, 63, 65, 200])
@pytest.mark.parametrize("form", ["rectangular", "triclinic", "nonperiodic"])
def test_tile_forms_match_the_oracle(n, form):
    rng = np.random.default_rng(n)
    sites = rng.permutation(343)[:n]  # a clump of 1.4 nm in the middle of the box
    ijk = np.stack([sites // 49, sites // 7 % 7, sites % 7], 1)
    pos = 2.3 + 0.2 * ijk + rng.uniform(-0.05, 0.05, (n, 3))
    q = [0.2 * (-1) ** i for i in range(n)]
    method = "CutoffNonPeriodic" if form == "nonperiodic" else "CutoffPeriodic"
    box = BOXES.get(form)
    s = ommb200.System()
    if box is not None:
        s.set_default_periodic_box_vectors(*box)
    nb = ommb200.NonbondedForce()
    nb.set_nonbonded_method(method)
    nb.set_cutoff_distance(RC)
    nb.set_use_dispersion_correction(False)
    exc = [(i, i + 1, 0.0, 0.2, 0.0) for i in range(0, n - 1, 5)]
    for i in range(n):
        s.add_particle(12.0)
        nb.add_particle(q[i], 0.2, 0.3 * (i % 3))
    for e in exc:
        nb.add_exception(*e)
    s.add_force(nb)
    ctx = ommb200.Context(s, systems.langevin(seed=1, step_size=0.001), precision="mixed")
    ctx.set_positions(pos)
    f_ref, e_ref = O.nonbonded(pos, q, [0.2] * n, [0.3 * (i % 3) for i in range(n)], exc,
                               method=method, cutoff=RC, box=box, use_dispersion_correction=False)
    st = ctx.get_state(forces=True, energy=True)
    # FP32 coordinates of up to 4 nm in the non-periodic form (1.2e-7 nm each) and neighbours as close
    # as 0.12 nm, whose forces go with r^-13: 13 * 1.4 * 1.2e-7 / 0.12 = 1.8e-5, energies alike
    if np.abs(f_ref).max() > 0:
        assert np.sqrt(((st.forces - f_ref) ** 2).sum() / (f_ref ** 2).sum()) < 1.8e-5
    assert abs(st.potential_energy - e_ref) < 1.8e-5 * abs(e_ref) + 2e-5 * n + 1e-5
    want = O.pair_set(pos, RC, np.diag([50.0] * 3) if box is None else box, [e[:2] for e in exc])
    got = ctx.debug_pair_list()
    key = lambda p: np.sort(np.sort(np.asarray(p).reshape(-1, 2), 1) @ np.array([n, 1]))  # noqa: E731
    assert np.array_equal(key(got), key(want))
