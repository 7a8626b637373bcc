"""UpdateProbs over the shapes of grid that choose its launch: the fixed-scratch form
against the allocating one where it takes more row pairs a block (and so more shared memory)
than that does; contexts of different grids in one process, in turn; and several row pairs
a block against the oracle.  All sums have one order, so every value must be equal
(tolerance: none)."""
import numpy as np
import pytest

from covidsim_b200 import abi, population, params as prm, sim
import oracle_py
from tests.helpers import snapshot, STATE_FIELDS

pytestmark = pytest.mark.gpu


def _world(ncw, nch, n_people=3000):
    grid = population.make_grid(nmcl=1)
    cell = min(1.0 / 120, 2.0 / max(ncw, nch))
    grid.update(ncw=ncw, nch=nch, cell_width=cell, cell_height=cell)
    pop = population.generate(n_people, grid, sigma=1.5, seed=3 + ncw)
    P, lk, hr = prm.build_params(grid, kernel_size=200000)
    P.LocalBeta = 0.9
    return pop, P, lk, hr


def _started(world, steps=12):
    """A Simulation `steps` timesteps into an epidemic."""
    s = sim.Simulation(*world)
    s.backend.begin_run(3, s.choose_seeds(3, 200))
    for k in range(steps):
        s.backend.step(k * world[1].ModelTimeStep)
    return s


def _same(a, b, where):
    for k in STATE_FIELDS:
        assert np.array_equal(a[k], b[k]), "%s: %s differs at %d entries" % (where, k, int(np.sum(a[k] != b[k])))


@pytest.mark.parametrize("ncw,nch", [(769, 311), (456, 648), (792, 632)])
def test_static_form_where_it_needs_more_shared_memory(ncw, nch):
    """One, two and one row pairs a block in the allocating form, two, three and three in the
    fixed-scratch one.  A small grid is brought up to date first, so that what an earlier call
    of this process enabled is not what the static call lives on."""
    small = _started(_world(200, 160), 0)
    small.backend.update_probs(0)
    ref, var = (_started(_world(ncw, nch)) for _ in range(2))
    var.backend.update_probs_static(0)
    ref.backend.update_probs(0)
    _same(snapshot(var.backend, var.pop), snapshot(ref.backend, ref.pop), "%d x %d" % (ncw, nch))
    for s in (small, ref, var):
        s.close()


@pytest.mark.parametrize("large,small", [((600, 600), (240, 240)), ((340, 260), (240, 240)), ((6000, 4), (5000, 4))])
def test_contexts_of_other_grids_take_turns(large, small):
    """More than 48 KB of shared memory a block each, the larger grid before, between and
    after calls of the smaller one: by direct calls, in a day graph captured after them, and
    from a replica made after them (above about 4,400 columns the unpacked kernel)."""
    a, b = _started(_world(*large)), _started(_world(*small))
    a.backend.update_probs(0)
    first = snapshot(a.backend, a.pop)
    for _ in range(2):
        b.backend.update_probs(0)
        a.backend.update_probs(0)
        _same(snapshot(a.backend, a.pop), first, "in turn")
    want, _ = a.run(5, 3, n_seed=100, probs_every_step=True, blocks=True)
    b.run(5, 3, n_seed=100, probs_every_step=True)
    a.backend.set_params(a.params)          # drops the day graph
    again, _ = a.run(5, 3, n_seed=100, probs_every_step=True, blocks=True)
    r = a.replica()
    other, _ = r.run(5, 3, n_seed=100, probs_every_step=True, blocks=True)
    for k in want:
        assert np.array_equal(want[k], again[k]) and np.array_equal(want[k], other[k]), k
    for s in (a, b, r):
        s.close()


@pytest.mark.parametrize("ncw,nch,n_people", [(120, 121, 500), (97, 201, 500), (241, 243, 700), (340, 259, 700)])
def test_several_row_pairs_a_block_match_the_oracle(ncw, nch, n_people):
    """Two, five, seven and eight row pairs a block, rows that are no multiple of theirs (the
    last block's pairs past the grid, the odd row among others), threads past the pairs, and
    with the last two more than 48 KB of shared memory."""
    world = _world(ncw, nch, n_people)
    pop, P = world[:2]
    sims = [sim.Simulation(*world), sim.Simulation(*world, backend=oracle_py.OracleBackend)]
    seeds = sims[0].choose_seeds(3, n_people // 4)
    for s in sims:
        s.backend.begin_run(3, seeds)
        for k in range(24):
            s.backend.infect_sweep(k * P.ModelTimeStep, 0)
            s.backend.incub_recovery_sweep(k * P.ModelTimeStep)
        s.backend.update_probs(0)
    a, b = (snapshot(s.backend, pop) for s in sims)
    assert not np.all(b["cell_tot_prob"] == 1.0)
    _same(a, b, "%d x %d" % (ncw, nch))
    # the tables' counts are those of the oracle too: the sweep after them draws from both alike
    for s in sims:
        s.backend.infect_sweep(24 * P.ModelTimeStep, 0)
    ca, cb = (abi.counters_to_dict(s.backend.counters()) for s in sims)
    assert ca == cb
    for s in sims:
        s.close()
