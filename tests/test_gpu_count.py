"""Count-only pair search (lm_count_pairs, LM_STEP_COUNT_PAIRS): the clustered stress workload.

The count must equal the size of cKDTree.query_pairs (golden lattice counts and boundary cases)
and the oracle's count on clustered positions whose cells hold thousands of microbes (the
shared-memory tiles of k_count_pairs), and the fused count step must count the pairs of exactly
the positions it advected.
"""

import numpy as np
import pytest

from conftest import golden

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine():
    from lagrangian_microbes_gb300 import engine as e
    return e


def clusters(rng, n_clusters, per, sigma, box=(200.0, 203.0, 25.0, 28.0)):
    cx = box[0] + (box[1] - box[0]) * rng.random(n_clusters)
    cy = box[2] + (box[3] - box[2]) * rng.random(n_clusters)
    sizes = np.maximum(1, (per * (np.arange(1, n_clusters + 1) ** -1.2) / np.mean(np.arange(1, n_clusters + 1) ** -1.2)).astype(int))
    lon = np.concatenate([c + sigma * rng.standard_normal(s) for c, s in zip(cx, sizes)])
    lat = np.concatenate([c + sigma * rng.standard_normal(s) for c, s in zip(cy, sizes)])
    return lon.astype(np.float32), lat.astype(np.float32)


def test_count_matches_ckdtree_lattices(engine, orc):
    g = golden("kdtree_lattice.npz")
    q = engine.PairQuery(0.01, 2)
    for (n, a, b, c, d), count in zip(g["configs"], g["counts"]):
        lons, lats = orc.lattice(int(n), a, b, c, d)
        assert q.count(lons.astype(np.float32), lats.astype(np.float32)) == count
    q.ctx.close()


def test_count_matches_ckdtree_boundary_cases(engine):
    g = golden("kdtree_cases.npz")
    for k in range(int(g["n_cases"])):
        X, r, p = g[f"c{k}_X"], float(g[f"c{k}_r"]), float(g[f"c{k}_p"])
        q = engine.PairQuery(r, p)
        assert q.count(X[:, 0], X[:, 1]) == len(g[f"c{k}_pairs"]), str(g[f"c{k}_name"])
        q.ctx.close()


@pytest.mark.parametrize("p", [2, 1, np.inf])
def test_count_dense_clusters_match_oracle(engine, orc, p):
    rng = np.random.default_rng(41)
    # Zipf-sized Gaussian clusters, sigma = 3 km: cores hold thousands of microbes per 0.01 deg cell
    lon, lat = clusters(rng, 40, 8000, 0.03)
    lon[::4001] = np.nan  # non-finite points are never paired
    q = engine.PairQuery(0.01, p)
    got = q.count(lon, lat)
    q.ctx.close()
    assert got == orc.count_pairs(lon, lat, 0.01, p)
    assert got > 1_000_000


def test_count_agrees_with_listed_pairs(engine, orc):
    rng = np.random.default_rng(43)
    lon, lat = clusters(rng, 12, 2500, 0.02)
    q = engine.PairQuery(0.01, 2)
    pi, pj = q.pairs(lon, lat)
    assert q.count(lon, lat) == pi.size == orc.count_pairs(lon, lat, 0.01, 2)
    q.ctx.close()


def test_fused_count_step_counts_the_advected_positions(engine, lm, orc, small_field):
    rng = np.random.default_rng(44)
    lon, lat = clusters(rng, 20, 3000, 0.03, box=(199.0, 202.0, 24.0, 27.0))
    sim = engine.Simulation(small_field, lon.astype(np.float64), lat.astype(np.float64),
                            np.ones(lon.size, np.int8), radius=0.01)
    totals = []
    for k in range(3):
        rec = sim.step(float(small_field.times[0]) + 3600.0 * k, 3600.0, 1, record=True, count_pairs=True)
        want = orc.count_pairs(rec["lon"][0], rec["lat"][0], 0.01, 2)
        st = sim.stats()
        assert st["pairs"] == want
        totals.append(want)
    assert sim.stats()["pairs_total"] == sum(totals)
    _, _, sp, _ = sim.state()
    assert (sp == 1).all()  # counting leaves the species alone
    sim.close()


@pytest.mark.parametrize("p", [2, 1, np.inf])
@pytest.mark.parametrize("per_cell", [40, 63, 64, 65, 300, 2500])
def test_count_over_leaves_of_dense_cells_matches_oracle(engine, orc, per_cell, p):
    """Cells around the size from which their members are counted by leaves of 32, with coincident
    microbes, pairs exactly one radius apart and sparse neighbours beside dense cells."""
    rng = np.random.default_rng(45 + per_cell)
    r = 0.01
    n = min(per_cell * 16, 12000)
    side = r * np.sqrt(n / per_cell)
    lon, lat = 200.0 + side * rng.random(n), 25.0 + side * rng.random(n)
    lon[:70], lat[:70] = lon[0], lat[0]  # one point, 70 times
    grid = np.arange(100)
    lon[100:200], lat[100:200] = 200.25 + 0.0078125 * (grid % 10), 25.25 + 0.0078125 * (grid // 10)
    lon[200:260] += 3 * side * rng.random(60)  # stragglers around the dense patch
    lon, lat = lon.astype(np.float32), lat.astype(np.float32)
    for radius in (r, 0.0078125, 0.0):
        q = engine.PairQuery(radius, p)
        assert q.count(lon, lat) == orc.count_pairs(lon, lat, radius, p), radius
        q.ctx.close()


def test_count_step_keeps_dense_ensembles_apart(engine, lm, orc, small_field):
    rng = np.random.default_rng(46)
    members, want = [], 0
    for n in (1, 3000, 33, 9000):
        lon, lat = 200.0 + 0.03 * rng.random(n), 25.0 + 0.03 * rng.random(n)
        members.append((lon, lat, np.ones(n, np.int8)))
    sim = engine.EnsembleSimulation(small_field, members, radius=0.01)
    rec = sim.step(float(small_field.times[0]), 3600.0, 1, record=True, count_pairs=True)
    for lon, lat in zip(sim.split(rec["lon"][0]), sim.split(rec["lat"][0])):
        want += orc.count_pairs(lon, lat, 0.01, 2)
    assert sim.stats()["pairs"] == want
    sim.close()


@pytest.mark.parametrize("size", [1, 2, 8, 9, 10, 33, 512, 513, 514, 1500])
def test_query_rows_of_every_list_length_are_in_order(engine, orc, size):
    """Clumps of `size` microbes that all pair with one another (lists of size - 1 partners: none, a
    slab row, a warp's shared row, beyond it) among scattered ones, in shuffled order."""
    rng = np.random.default_rng(47 + size)
    lon = np.concatenate([200.1 + 0.004 * rng.random(size), 200.5 + 0.004 * rng.random(size), 200 + rng.random(3000)])
    lat = np.concatenate([25.1 + 0.004 * rng.random(size), 25.5 + 0.004 * rng.random(size), 25 + rng.random(3000)])
    order = rng.permutation(lon.size)
    lon, lat = lon[order].astype(np.float32), lat[order].astype(np.float32)
    lon[0] = np.nan
    q = engine.PairQuery(0.01, 2)
    pi, pj = q.pairs(lon, lat)
    assert q.count(lon, lat) == pi.size
    q.ctx.close()
    oi, oj = orc.pairs(lon, lat, 0.01, 2)
    np.testing.assert_array_equal(pi, oi)
    np.testing.assert_array_equal(pj, oj)


def test_count_at_the_inner_edge_of_the_float32_band(engine):
    """A radius and a distance whose place in the band around the radius comes out 5 units in the last place below 1, so
    that the sum of the places of a tile falls short of the whole number it stands for."""
    r, d = 0.007813882993826751, np.float32(0.007813866)
    assert float(d) < r
    far = np.array([0.999 * d] * 5 + [d] + [1.003 * d] * 26, np.float32)
    lon = np.concatenate([np.zeros(2048, np.float32), np.tile(far, 16)])
    lat = np.zeros(lon.size, np.float32)
    inside = int((far <= r).sum()) * 16
    among = lambda m: m * (m - 1) // 2  # each of the two groups spans less than the radius
    want = among(2048) + 2048 * inside + among(16 * far.size)
    q = engine.PairQuery(r, np.inf)
    assert q.count(lon, lat) == want
    q.ctx.close()


def test_lists_beyond_32_bit_offsets_are_refused_and_the_context_stays_usable(engine, lm):
    """70,000 microbes in one place have 4.9e9 list entries, more than the area of long lists can ever hold: an error, where
    the area would be enlarged and the search repeated for ever. They can still be counted."""
    n = 70_000
    lon, lat = np.full(n, 200.5, np.float32), np.full(n, 25.5, np.float32)
    q = engine.PairQuery(0.01, 2)
    with pytest.raises(lm.LMError) as failed:
        q.pairs(lon, lat)
    assert failed.value.code == lm._lib.LM_ERR_ROUND_CAP
    assert q.count(lon, lat) == n * (n - 1) // 2
    pi, pj = q.pairs(lon[:300], lat[:300])
    assert pi.size == 300 * 299 // 2 and (pi < pj).all()
    q.ctx.close()
