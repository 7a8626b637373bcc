"""The whole-timestep path (cs_gpu_step: one scan ahead of the infections, the infections
beside the transitions, all list moves at the end) against the sweeps called one by one and
the oracle, state for state (tolerance: none), where the two forms could part: people
infected and turning infectious in the same timestep (a latent period of a tenth of a step),
and dying or recovering in it too (an infectious period of no steps), cells with more moves
in a step than a warp's batch of 32, whole timesteps and single sweeps in turn, and false
positives switched on and off between steps."""
import numpy as np
import pytest

from covidsim_b200 import abi, population, params as prm, sim
import oracle_py
from tests.helpers import snapshot, check_lists, STATE_FIELDS

pytestmark = pytest.mark.gpu


def _world(n_people, cells, latent, infectious):
    grid = population.make_grid(nmcl=2)
    grid.update(ncw=cells, nch=cells, cell_width=1.0 / 120, cell_height=1.0 / 120)
    pop = population.generate(n_people, grid, sigma=1.0, seed=11)
    P, lk, hr = prm.build_params(grid, kernel_size=200000)
    P.LocalBeta = 2.0
    if latent is not None:
        P.LatentPeriod = latent
    if infectious is not None:
        P.InfectiousPeriod = infectious
    return pop, P, lk, hr


def _same(a, b, where):
    for k in STATE_FIELDS:
        assert np.array_equal(a[k], b[k]), "%s: %s differs at %d entries" % (where, k, int(np.sum(a[k] != b[k])))


@pytest.mark.parametrize("n_people,cells,latent,infectious,n_seed", [
    (3000, 1, None, None, 900), (6000, 4, 0.02, None, 300), (6000, 4, 0.02, 0.1, 300), (20000, 30, 0.3, 1.0, 4000)])
def test_step_matches_single_sweeps_and_oracle(n_people, cells, latent, infectious, n_seed):
    pop, P, lk, hr = _world(n_people, cells, latent, infectious)
    whole, single = sim.Simulation(pop, P, lk, hr), sim.Simulation(pop, P, lk, hr)
    orac = sim.Simulation(pop, P, lk, hr, backend=oracle_py.OracleBackend)
    seeds = whole.choose_seeds(5, n_seed)
    for s in (whole, single, orac):
        s.backend.begin_run(5, seeds)
    for k in range(48):
        t = k * P.ModelTimeStep
        if k in (16, 24):   # the false-positive path, and back
            for s in (whole, single, orac):
                q = abi.cs_params.from_buffer_copy(P)
                q.FalsePositiveRate = 0.2 if k == 16 else 0.0
                s.backend.set_params(q)
        if k % 7 == 6:      # whole timesteps and single sweeps of one context in turn
            whole.backend.infect_sweep(t, 0)
            whole.backend.incub_recovery_sweep(t)
        else:
            whole.backend.step(t, 0)
        for s in (single, orac):
            s.backend.infect_sweep(t, 0)
            s.backend.incub_recovery_sweep(t)
        if k == 30:
            for s in (whole, single, orac):
                s.backend.seed_infections(t, np.arange(0, n_people, 50, dtype=np.int32))
        if k % 5 == 0 or k in (16, 17, 24, 30, 31, 47):
            b = snapshot(orac.backend, pop)
            _same(snapshot(whole.backend, pop), b, "step %d" % k)
            _same(snapshot(single.backend, pop), b, "sweeps %d" % k)
    check_lists(b, pop)
    cs = [abi.counters_to_dict(s.backend.counters()) for s in (whole, single, orac)]
    assert cs[0] == cs[1]
    # the mid-run seeding names people already infected; the oracle measures radii from the
    # last person named, the library from the last one it infects
    for k in set(cs[0]) - {"sumRad2_q", "maxRad2_bits"}:
        assert cs[0][k] == cs[2][k], k
    for s in (whole, single, orac):
        s.close()


@pytest.mark.parametrize("n_people,cells,n_seed", [(2001, 4, 40), (40000, 30, 16000)])
def test_lanes_per_contact_by_the_load(n_people, cells, n_seed):
    """A grid of eight blocks has 256 groups of eight lanes, so that more than 5,120 infectors
    take groups of four: the states are those of every number that can be set."""
    pop, P, lk, hr = _world(n_people, cells, 0.3, None)
    sims = {lanes: sim.Simulation(pop, P, lk, hr) for lanes in (0, 2, 4, 8, 16)}
    seeds = sims[0].choose_seeds(9, n_seed)
    for lanes, s in sims.items():
        s.backend.set_grid(8 if lanes == 0 else 592)
        if lanes:
            s.backend.set_spatial_lanes(lanes)
        s.backend.begin_run(9, seeds)
    most, before = 0, 0
    for k in range(16):
        for s in sims.values():
            s.backend.step(k * P.ModelTimeStep, 0)
        now = int(sims[0].backend.counters().work_infectors)
        most, before = max(most, now - before), now
    assert (most > 5120) == (n_people == 40000)
    want = snapshot(sims[8].backend, pop)
    for lanes, s in sims.items():
        _same(snapshot(s.backend, pop), want, "%d lanes" % lanes)
        assert abi.counters_to_dict(s.backend.counters()) == abi.counters_to_dict(sims[8].backend.counters())
    for s in sims.values():
        s.close()


@pytest.mark.parametrize("device_loop", [False, True])
def test_households_left_by_an_infect_sweep_alone(device_loop):
    """The false cases of an infection sweep leave flagged households to the next transitions,
    also when those are a whole timestep's or the device run loop's, with false positives off."""
    pop, P, lk, hr = _world(6000, 4, None, None)
    whole, single = sim.Simulation(pop, P, lk, hr), sim.Simulation(pop, P, lk, hr)
    orac = sim.Simulation(pop, P, lk, hr, backend=oracle_py.OracleBackend)
    sims, dt = (whole, single, orac), P.ModelTimeStep
    on, off = abi.cs_params.from_buffer_copy(P), abi.cs_params.from_buffer_copy(P)
    on.FalsePositiveRate = 0.5
    iv = abi.cs_interventions()
    iv.CaseIsolationPolicyDuration = iv.HQuarantinePolicyDuration = 1000.0
    seeds = whole.choose_seeds(5, 100)   # few enough that the day's end recomputes no probabilities
    for s in sims:
        s.backend.begin_run(5, seeds)
        s.backend.set_interventions(iv)
        for k in range(12):
            s.backend.step(k * dt, 0)
        s.backend.set_params(on)
        s.backend.infect_sweep(12 * dt, 0)
        s.backend.set_params(off)
    before = snapshot(orac.backend, pop)
    steps = int(P.TimeStepsPerDay) if device_loop else 3
    for s in sims:
        if s is whole and device_loop:
            s.backend.run_device(1, sim.run_policy(None, pop.num_place_types))
            continue
        for k in range(0 if device_loop else 13, steps if device_loop else 16):
            if s is whole:
                s.backend.step(k * dt, 0)
            else:
                s.backend.infect_sweep(k * dt, 0)
                s.backend.incub_recovery_sweep(k * dt)
    want = snapshot(orac.backend, pop)
    assert not np.array_equal(before["quar_start_time"], want["quar_start_time"])
    _same(snapshot(single.backend, pop), want, "sweeps")
    _same(snapshot(whole.backend, pop), want, "whole timesteps")
    for s in sims:
        s.close()


def test_the_choice_of_lanes_by_the_load_can_be_had_back():
    pop, P, lk, hr = _world(2001, 4, 0.3, None)
    a = sim.Simulation(pop, P, lk, hr)
    b = a.replica()
    batch = sim.Batch([b])
    for be in (a.backend, batch):
        be.set_spatial_lanes(4)
        be.set_spatial_lanes(0)
        for lanes in (-1, 1, 3, 32):
            with pytest.raises(abi.CovidSimError):
                be.set_spatial_lanes(lanes)
    seeds = a.choose_seeds(9, 100)
    for s in (a, b):
        s.backend.begin_run(9, seeds)
    for k in range(8):
        a.backend.step(k * P.ModelTimeStep, 0)
        batch.step(k * P.ModelTimeStep, 0)
    _same(snapshot(a.backend, pop), snapshot(b.backend, pop), "alone and in a batch")
    batch.close()
    a.close()
    b.close()


def test_counters_match_the_oracle_before_any_mid_run_seeding():
    """Every counter, the radii of infection (summed by warps beside the transitions) too."""
    for n_people, cells, latent, n_seed in ((6000, 4, 0.02, 300), (20000, 30, 0.3, 1000)):
        pop, P, lk, hr = _world(n_people, cells, latent, None)
        sims = [sim.Simulation(pop, P, lk, hr), sim.Simulation(pop, P, lk, hr, backend=oracle_py.OracleBackend)]
        seeds = sims[0].choose_seeds(5, n_seed)
        for s in sims:
            s.backend.begin_run(5, seeds)
            for k in range(29):
                s.backend.step(k * P.ModelTimeStep, 0)
        a, b = (abi.counters_to_dict(s.backend.counters()) for s in sims)
        assert b["sumRad2_q"] > 0 and b["maxRad2_bits"] > 0
        assert a == b
        for s in sims:
            s.close()


def test_parameters_beyond_their_tables():
    """Households whose size for the kernel lies past its table read what the parameter block
    holds there, as the oracle does; a sweep at a time long before its infectors turned
    infectious reads nothing outside the block."""
    pop, P, lk, hr = _world(2001, 4, None, None)
    pop.hh_nhr = np.full_like(pop.hh_nhr, 300)          # entry 299: entry 289 of the profile behind it
    q = abi.cs_params.from_buffer_copy(P)
    q.infectiousness[289] = 0.7
    q.LocalBeta = 0.5
    sims = [sim.Simulation(pop, q, lk, hr), sim.Simulation(pop, q, lk, hr, backend=oracle_py.OracleBackend)]
    seeds = sims[0].choose_seeds(5, 60)
    for s in sims:
        s.backend.begin_run(5, seeds)
        for k in range(32):
            s.backend.step(k * q.ModelTimeStep, 0)
    a, b = (snapshot(s.backend, pop) for s in sims)
    _same(a, b, "large households")
    assert np.sum(b["infect_type"] % abi.CONST["CS_INFECT_TYPE_MASK"] == 1) > 20     # infections in households
    g = sims[0].backend
    for k in range(32, 240):
        g.step(k * q.ModelTimeStep, 0)
    g.infect_sweep(0.0, 0)
    g.incub_recovery_sweep(0.0)
    g.sync()
    check_lists(snapshot(g, pop), pop)
    for s in sims:
        s.close()
