"""The assignment of people to places at the edges of the warp-wide nearest-place search:
choices among one place and among a whole warp's worth, fewer places than are looked for, one
bucket, a strip of cells (rings cut off at the grid's edge), rings of more than a warp's
columns, one round and none before the last, and attendee counts at which a warp looks
through one person or several.  Against the sequential oracle, array for array (bit-exact)."""
import numpy as np
import pytest

from covidsim_b200 import population

pytestmark = pytest.mark.gpu

WORLDS = {
    "one_cell": (400, dict(ncw=1, nch=1), [1, 2, 32, 31], 6, {}),
    "strip": (3000, dict(ncw=1, nch=40), [32, 1, 3, 24], 6, dict(sigma=1.5)),
    "sparse_wide": (2500, dict(ncw=60, nch=60), [2, 32, 32, 32], 1, dict(sigma=3.0)),
    "last_round_only": (6000, dict(ncw=12, nch=8), [5, 32, 1, 24], 0, {}),
    "several_a_warp": (90000, dict(ncw=24, nch=24), [3, 3, 32, 24], 3, dict(blobs=3, blob_share=0.6)),
}


@pytest.mark.parametrize("name", sorted(WORLDS))
def test_places_match_oracle(name, monkeypatch):
    import oracle_py
    n, cells, nearest, rounds, kw = WORLDS[name]
    monkeypatch.setattr(population, "PLACE_NEAREST", nearest)
    grid = population.make_grid(nmcl=2)
    grid.update(cells, cell_width=1.0 / 120, cell_height=1.0 / 120)
    g = population.generate_on_device(n, grid, rounds=rounds, seed=31, **kw)
    o = oracle_py.setup_population(n, grid, rounds=rounds, seed=31, **kw)
    for k in population._ARRAYS:
        assert np.array_equal(getattr(g, k), getattr(o, k)), "%s differs" % k
    for t, (pg, po) in enumerate(zip(g.places, o.places)):
        for k in population._PLACE_ARRAYS:
            assert np.array_equal(pg[k], po[k]), "place type %d %s differs" % (t, k)
    assert g.setup_info["forced"] == o.setup_info["forced"]
