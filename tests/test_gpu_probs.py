"""UpdateProbs and the proposal tables it rebuilds, on the GPU against the oracle, at the
edges of the kernels' tiles: grids whose columns leave a remainder of the 8 columns a
thread owns and of the 16-column windows, odd numbers of rows (the last row of the packed
pairs stands alone), several row chunks, and proposal blocks from one cell each (more
than 32 rows a block of threads, more targets than a tile) to all cells in one.  Both
sides add in the same order, so every value must be equal (tolerance: none)."""
import numpy as np
import pytest

from covidsim_b200 import population, params as prm, sim
import oracle_py
from tests.helpers import snapshot, STATE_FIELDS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ncw,nch,block_cells,n_people", [
    (1, 1, 0, 60), (7, 3, 1, 300), (8, 33, 0, 2000), (17, 32, 2, 2500), (33, 65, 1, 6000), (70, 64, 1, 9000),
    (61, 7, 61, 3000), (129, 5, 0, 4000)])
def test_update_probs_matches_oracle(ncw, nch, block_cells, n_people):
    grid = population.make_grid(nmcl=2)
    grid.update(ncw=ncw, nch=nch, cell_width=1.0 / 120, cell_height=1.0 / 120)
    pop = population.generate(n_people, grid, sigma=1.5, seed=5 + ncw)
    P, lk, hr = prm.build_params(grid, kernel_size=200000)
    P.block_cells = block_cells
    P.LocalBeta = 0.9
    sims = [sim.Simulation(pop, P, lk, hr), sim.Simulation(pop, P, lk, hr, backend=oracle_py.OracleBackend)]
    seeds = sims[0].choose_seeds(3, max(1, n_people // 20))
    for s in sims:
        s.backend.begin_run(3, seeds)
    for k in range(60):
        for s in sims:
            if k % 20 == 10:
                s.backend.update_probs(0)
            s.backend.infect_sweep(k * P.ModelTimeStep, 0)
            s.backend.incub_recovery_sweep(k * P.ModelTimeStep)
        if k % 20 in (10, 19):
            a, b = (snapshot(s.backend, pop) for s in sims)
            for f in STATE_FIELDS:
                assert np.array_equal(a[f], b[f]), "step %d: %s differs at %d entries" % (k, f, int(np.sum(a[f] != b[f])))
    for s in sims:
        s.close()
