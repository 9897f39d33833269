"""The volume gather's tensor-core tiles (tiles.cuh) against the list form and the oracle."""
import ctypes

import numpy as np
import pytest

import helpers as H

pytestmark = pytest.mark.gpu


def _bent(pos):
    p = pos.astype(np.float64)
    a = 0.4 * p[:, 0]
    return np.stack([p[:, 0] * 1.1, np.cos(a) * p[:, 1] - np.sin(a) * p[:, 2],
                     np.sin(a) * p[:, 1] + np.cos(a) * p[:, 2]], 1).astype(np.float32)


def _one_iteration(solver, scene, lanes=None, positions=None, **kw):
    """One substep of one iteration from bent positions; ``lanes`` forces the gather's form."""
    scen = H.scenes.Scenario(scene, [], iters=1, shape=False, **kw)
    scen.setup(solver)
    solver.step()
    solver.reset()
    solver.set_positions(_bent(scene["pos"]) if positions is None else positions)
    if lanes is not None:
        solver.lib.xpbd_b200_set_volume_lanes.argtypes = [ctypes.c_int] * 2
        solver.lib.xpbd_b200_set_volume_lanes(0, lanes)
    solver.step()
    if lanes is not None:
        solver.lib.xpbd_b200_set_volume_lanes(0, 0)
    return solver.positions()


# components below, at and above the tile size and its remainders; several components; short
# lists (none in tiles); more columns than one slab holds and groups of over 32 mask blocks
CASES = [
    ((63,), 8, {}, False), ((64,), 8, {}, True), ((65,), 8, {}, True), ((128,), 8, {}, True),
    ((129,), 8, {}, True), ((300, 70, 1000), 8, {}, True), ((2500,), 8, dict(max_members=16), False),
    ((2500,), 8, dict(max_members=24), True), ((3000,), 12, dict(max_members=128), True),
    ((9000,), 12, dict(ring_k=4, max_members=200), True), ((4000,), 8, dict(max_members=2048, leader_min_hop=3), None),
]


@pytest.mark.parametrize("sizes,knn,kw,in_tiles", CASES)
def test_tile_gather_matches_lists_and_oracle(sizes, knn, kw, in_tiles):
    """A record is rounded to 2^-23 of the largest of its kind (M at most about 1, M (c - o) at
    most the tile's size), so a mean of records differs from the list form's by at most 6 x
    2^-23 of the diagonal, 0.6 of which moves the position; plus FP32 rounding of the position."""
    scene = H.scenes.merge_scenes([H.scenes.make_scene(n, 7 + k, knn=knn, centre=(3.0 * k, 0.0, 0.0))
                                   for k, n in enumerate(sizes)])
    lib, orc = H.b200(), H.oracle()
    tile = _one_iteration(lib, scene, 0, **kw)
    tiles, rows = lib.ints("gather_tiles")
    assert rows + (0 if tiles == 0 else sum(sizes) - rows) == sum(sizes)
    if in_tiles is not None:
        assert (tiles > 0) == in_tiles
    lists = _one_iteration(lib, scene, 4, **kw)
    ref = _one_iteration(orc, scene, **kw)
    lib.destroy()
    orc.destroy()
    diag = H.scenes.bbox_diagonal(ref)
    assert H.max_err_over_diag(tile, lists, diag) < 0.6 * 6 * 2.0 ** -23 + 2.0 ** -23
    assert H.max_err_over_diag(tile, ref, diag) < H.TOL_1STEP


@pytest.mark.parametrize("value", [np.nan, np.inf, 1e20, 50.0])
def test_tile_gather_with_a_position_gone_astray(value):
    """One Gaussian far off or not finite: every row comes out as from the lists."""
    scene = H.scenes.make_scene(1500, 5)
    pos = _bent(scene["pos"])
    pos[700, 1] = value
    lib = H.b200()
    tile = _one_iteration(lib, scene, 0, positions=pos)
    lists = _one_iteration(lib, scene, 4, positions=pos)
    lib.destroy()
    np.testing.assert_array_equal(np.isfinite(tile), np.isfinite(lists))
    ok = np.isfinite(lists).all(1) & (np.abs(lists).max(1) < 10.0)
    diag = H.scenes.bbox_diagonal(lists[ok])
    assert H.max_err_over_diag(tile[ok], lists[ok], diag) < 0.6 * 6 * 2.0 ** -23 + 2.0 ** -23
