"""Guided renders on every route a wave can take: a path per thread or per four lanes (small images)
and a launch per bounce (large ones, and any size in measurement mode).  Each route against the CPU
integrator, and the routes against each other: images, path depths and counters bit for bit, the
SD-tree's sums and topology, the hash grid's cells with their quadtrees."""
import numpy as np
import pytest

from rtlib_b200 import scenes

pytestmark = pytest.mark.gpu

BOX = ((-0.005,) * 3, (1.005,) * 3)
ROOMS = ((-0.005,) * 3, (14.005, 4.005, 10.005))


def _scene(kind, w, h):
    if kind == "flat":
        return scenes.cornell_box(w, h), BOX
    return scenes.occluded_rooms(w, h, n_objects=20, n_lights=64, seed=5, sphere_level=0), ROOMS


def _tree_render(cuda, kind, w, h, flags, waves, budget, ratio, depth):
    from rtlib_b200.sdtree import SDTree, SDTreeController
    from rtlib_b200.tracer import Tracer
    sc, box = _scene(kind, w, h)
    tree = SDTree(*box, fraction=0.5)
    ctrl = SDTreeController(tree, budget, iteration_for_built=0, ratio_for_budget=ratio, samples_per_launch=1)
    tr = Tracer(sc, cuda, max_depth=depth, width=w, height=h, seed=5)
    tr.set_timing(waves)
    ctrl.start()
    tr.render_guided(tree, ctrl, flags, samples_per_launch=1)
    assert tree.status() == 0
    return tr, tree


def _grid_render(cuda, kind, w, h, flags, waves, budget, depth, keying=1, max_launches=1 << 30):
    from rtlib_b200.hashgrid import HashGrid, MortonQuadTreeController, MortonQuadTrees
    from rtlib_b200.tracer import Tracer
    sc, box = _scene(kind, w, h)
    bounds, slots = ((16, 16, 16), 4096) if kind == "flat" else ((64, 16, 48), 1 << 15)
    grid = HashGrid(*box, bounds, slots, keying=keying)
    trees = MortonQuadTrees(slots, level=4, fraction=0.5)
    ctrl = MortonQuadTreeController(trees, budget, iteration_for_built=1, iteration_for_locate=0, ratio_for_budget=0.5,
                                    samples_per_launch=1)
    tr = Tracer(sc, cuda, max_depth=depth, width=w, height=h, seed=5)
    tr.set_timing(waves)
    grid.clear()
    ctrl.start()
    tr.render_grid_guided(grid, trees, ctrl, flags, max_launches=max_launches)
    assert grid.status() == 0 and trees.status() == 0
    return tr, grid, trees


def _cells(grid, trees):
    """Keys in order, and each key's building leaves and pyramid."""
    cur = grid.export()
    slot = np.flatnonzero(cur)
    slot = slot[np.argsort(cur[slot])]
    leaves, pyramid = trees.export()
    n = trees.num_cells
    return cur[slot], leaves.reshape(n, -1)[slot], pyramid.reshape(n, -1)[slot]


def _same_render(a, b):
    np.testing.assert_array_equal(a.image64().cpu().numpy(), b.image64().cpu().numpy())
    np.testing.assert_array_equal(a.path_depths().cpu().numpy(), b.path_depths().cpu().numpy())
    assert a.counters() == b.counters() and a.stats() == b.stats()


# four lanes a path; a lane a path; both sides of the limit for RIS (5 CTAs of 128 paths per SM); a launch
# per bounce (past 7 of them); and scenes that rays walk a hierarchy in
ROUTES = [("flat", 48, 48), ("flat", 149, 80), ("flat", 148 * 5, 128), ("flat", 148 * 5, 129), ("flat", 148 * 7, 129),
          ("rooms", 64, 36), ("rooms", 300, 200)]


@pytest.mark.parametrize("kind,w,h", ROUTES)
@pytest.mark.parametrize("flags", [0, 1, 3])
def test_tree_guided_routes_agree(cuda, kind, w, h, flags):
    """Passes that record, record and sample, and only sample (the budget's second half)."""
    (a, ta), (b, tb) = (_tree_render(cuda, kind, w, h, flags, waves, 15, 0.5, 7) for waves in (False, True))
    _same_render(a, b)
    for ea, eb in zip((ta.export(True), ta.export(False)), (tb.export(True), tb.export(False))):
        assert ea.topology == eb.topology
        np.testing.assert_array_equal(ea.scalars, eb.scalars)
        np.testing.assert_array_equal(ea.dsums, eb.dsums)


@pytest.mark.parametrize("kind,w,h", ROUTES)
@pytest.mark.parametrize("flags", [1, 3])
def test_grid_guided_routes_agree(cuda, kind, w, h, flags):
    """Passes that locate, record, record and sample, and only sample.  Concurrent inserts claim slots
    in any order: cells are compared by key."""
    (a, *ga), (b, *gb) = (_grid_render(cuda, kind, w, h, flags, waves, 15, 7) for waves in (False, True))
    _same_render(a, b)
    for x, y in zip(_cells(*ga), _cells(*gb)):
        np.testing.assert_array_equal(x, y)


def _close(tr, want, rel_mse=2e-3, frac=0.97):
    got = tr.image().cpu().numpy()
    rel = np.abs(got - want) / np.maximum(np.abs(want), 1e-2)
    assert np.mean((got - want) ** 2) < rel_mse * np.mean(want ** 2)
    assert (rel < 1e-3).all(axis=2).mean() > frac


# (the bounds of the small guided renders against the oracle in test_tracer_gpu.py)
@pytest.mark.parametrize("kind,w,h,budget,flags", [("flat", 48, 48, 31, 1), ("rooms", 48, 27, 7, 3), ("flat", 148 * 7, 129, 3, 1)])
def test_tree_guided_waves_match_oracle(cuda, oracle, kind, w, h, budget, flags):
    from oracle.oracle import OracleRenderer
    depth = 8
    tr, tree = _tree_render(cuda, kind, w, h, flags, True, budget, 1.0, depth)
    sc, box = _scene(kind, w, h)
    ot = oracle.sdtree(*box)
    r = OracleRenderer(oracle, sc, width=w, height=h, max_depth=depth, num_candidates=32, fraction=0.5, seed=5)
    r.render_guided(ot, budget, ratio_for_budget=1.0, base_flags=flags)
    assert tr.stats()["samples"] == r.samples
    _close(tr, r.image())
    eg, eo = tree.export(True), ot.export(True)
    if kind == "flat":
        assert eg.topology == eo.topology
        close = np.abs(eg.dsums - eo.dsums) <= 1e-3 * np.abs(eo.dsums) + 1e-2
        assert close.mean() > 0.9
    # a separated path moves its whole contribution; few paths carry much of the rooms' light
    assert abs(eg.dsums.sum() - eo.dsums.sum()) < (1e-2 if kind == "flat" else 1e-1) * eo.dsums.sum()


# (the rooms: test_occluded_grid_guided_ris_matches_oracle, whose route equals the waves)
@pytest.mark.parametrize("kind,w,h,budget,flags", [("flat", 48, 48, 31, 1), ("flat", 148 * 7, 129, 3, 1)])
def test_grid_guided_waves_match_oracle(cuda, oracle, kind, w, h, budget, flags):
    from oracle.oracle import OracleGrid, OracleRenderer
    depth = 8
    tr, grid, trees = _grid_render(cuda, kind, w, h, flags, True, budget, depth)
    sc, box = _scene(kind, w, h)
    bounds, slots = ((16, 16, 16), 4096) if kind == "flat" else ((64, 16, 48), 1 << 15)
    og = OracleGrid(oracle, *box, bounds, slots, keying=1, level=4, fraction=0.5)
    r = OracleRenderer(oracle, sc, width=w, height=h, max_depth=depth, num_candidates=32, seed=5)
    r.render_grid_guided(og, budget, iteration_for_built=1, iteration_for_locate=0, ratio_for_budget=0.5, base_flags=flags)
    assert tr.stats()["samples"] == r.samples and og.status == 0
    _close(tr, r.image())
    np.testing.assert_array_equal(_cells(grid, trees)[0], np.sort(og.cur[og.cur != 0]))
