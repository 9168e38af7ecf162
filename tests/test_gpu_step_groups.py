"""Context.step in groups and single steps: any split of a run into calls gives the same trajectory
as the launches one by one, bit for bit; a barostat, whose accepted moves drop the captured graphs,
too."""
import numpy as np
import pytest

import ommb200
from ommb200 import synth, systems

pytestmark = pytest.mark.gpu


def _water(**kw):
    w = synth.water_box(216, 1.9, (6, 6, 6), seed=3)
    ctx = ommb200.Context(systems.water_system(w), systems.langevin(seed=5), **kw)
    ctx.set_positions(w.positions)
    return ctx


def _water_chain(**kw):  # the reciprocal part as a launch chain, beside the rebuilds
    return _water(pme_bricks=0, **kw)


def _chain(**kw):
    ch = synth.chain(150, seed=2)
    ctx = ommb200.Context(systems.chain_system(ch), systems.langevin(seed=5, step_size=0.001), **kw)
    ctx.set_positions(ch.positions)
    return ctx


@pytest.mark.parametrize("make", [_water, _water_chain, _chain])
@pytest.mark.parametrize("calls", [[47], [20, 20, 7], [1] * 47, [19, 21, 7], [46, 1], [3, 40, 4]])
def test_step_groups_give_one_trajectory(make, calls):
    res = []
    for graph, split in ((False, [47]), (True, calls)):
        ctx = make(use_cuda_graph=graph)
        ctx.set_velocities_to_temperature(300.0, seed=1)
        for k in split:
            ctx.step(k)
        st = ctx.get_state(positions=True, velocities=True, forces=True)
        assert st.step_count == 47
        res.append(st)
        ctx.close()
    assert np.array_equal(res[0].positions, res[1].positions)
    assert np.array_equal(res[0].velocities, res[1].velocities)
    assert np.array_equal(res[0].forces, res[1].forces)


@pytest.mark.parametrize("frequency,steps", [(1, 6), (7, 30), (25, 60), (130, 300)])
def test_barostat_graphs_match_the_stream_path(frequency, steps):
    out = []
    for graph in (False, True):
        w = synth.water_box(343, 2.25, (7, 7, 7), seed=4)
        s = systems.water_system(w)
        bar = ommb200.MonteCarloBarostat(1.0, 300.0, frequency)
        bar.set_random_number_seed(9)
        s.add_force(bar)
        ctx = ommb200.Context(s, systems.langevin(seed=5), use_cuda_graph=graph)
        ctx.set_positions(w.positions)
        ctx.set_velocities_to_temperature(300.0, seed=1)
        ctx.step(steps)
        st = ctx.get_state(positions=True)
        out.append((st.positions, st.periodic_box_vectors, ctx.barostat_stats()["accepted"]))
        ctx.close()
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
    assert out[0][2] == out[1][2]
