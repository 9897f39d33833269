"""The switches between the step's forms: which kernels a step runs, and what comes out."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest

import helpers as H

pytestmark = pytest.mark.gpu

ITERS = 3


def _lanes(solver, solve, gather):
    solver.lib.xpbd_b200_set_volume_lanes.argtypes = [ctypes.c_int] * 2
    solver.lib.xpbd_b200_set_volume_lanes(solve, gather)


def _tuning(solver):
    t = np.zeros(7, np.float32)
    solver.lib.xpbd_b200_tuning.argtypes = [ctypes.c_void_p]
    solver.lib.xpbd_b200_tuning(t.ctypes.data)
    return t


def _fused(solver, mode):
    solver.lib.xpbd_b200_set_fused.argtypes = [ctypes.c_int]
    solver.lib.xpbd_b200_set_fused(mode)


@pytest.fixture
def lib():
    solver = H.b200()
    yield solver
    _lanes(solver, 0, 0)
    _fused(solver, 0)
    solver.destroy()


def _mixed(solver):
    """Rows in tiles and, in a small component, rows in the list form."""
    scene = H.scenes.merge_scenes([H.scenes.make_scene(300, 1), H.scenes.make_scene(40, 2, centre=(4.0, 0.0, 0.0))])
    H.scenes.Scenario(scene, [], iters=ITERS, shape=False).setup(solver)
    return scene


def test_lanes_set_after_a_step_take_effect(lib):
    """Automatic: a launch for the tiles and one for the lists; four lanes: the lists alone."""
    _mixed(lib)
    lib.step()
    tiles, rows = lib.ints("gather_tiles")
    assert tiles > 0 and rows == 40
    both = _tuning(lib)[4]
    _lanes(lib, 0, 4)
    lib.step()
    assert _tuning(lib)[4] == both - ITERS
    _lanes(lib, 0, 0)
    lib.step()
    assert _tuning(lib)[4] == both


def test_lists_asked_for_leave_the_fused_form(lib):
    """The fused launch runs the tiles, so it does not stand in for the list form."""
    _mixed(lib)
    _fused(lib, 1)
    lib.step()
    assert _tuning(lib)[0] == 1.0
    _lanes(lib, 0, 4)
    lib.step()
    assert _tuning(lib)[0] == 0.0


SMALL = """
import ctypes, sys
sys.path.insert(0, sys.argv[1])
import numpy as np
import helpers as H
lib, t = H.b200(), np.zeros(7, np.float32)
lib.raw.xpbd_b200_set_fused(1)
H.scenes.Scenario(H.scenes.make_scene(50, 1), []).setup(lib)
lib.step()
lib.raw.xpbd_b200_tuning.argtypes = [ctypes.c_void_p]
lib.raw.xpbd_b200_tuning(t.ctypes.data)
lib.destroy()
print(int(t[0]), int(t[4]))
"""


def test_fused_form_without_tiles():
    """A scene too small for tiles, the first of its process, takes the fused launch too."""
    tests = os.path.dirname(os.path.abspath(__file__))
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([H.ROOT, os.environ.get("PYTHONPATH", "")]))
    r = subprocess.run([sys.executable, "-c", SMALL, tests], capture_output=True, text=True, timeout=300, env=env)
    assert r.returncode == 0, r.stderr
    assert r.stdout.split() == ["1", "1"]


def _one_iteration(positions, scene, lanes, members=32):
    """One substep of one volume iteration from ``positions``, the gather's lanes set before it."""
    solver = H.b200()
    H.scenes.Scenario(scene, [], iters=1, shape=False, max_members=members).setup(solver)
    solver.set_constraints(distance=False, shape=False, angle=False, volume=True)
    _lanes(solver, 0, lanes)
    solver.step()
    solver.reset()
    solver.set_positions(positions)
    solver.step()
    tiles = solver.ints("gather_tiles")
    _lanes(solver, 0, 0)
    out = solver.positions()
    solver.destroy()
    return out, tiles


POSES = {
    "half pressed flat": lambda p: np.where(p[:, :1] > 0.0, p * [1.0, 1.0, 0.05], p),
    "half pressed": lambda p: np.where(p[:, :1] > 0.0, p * [1.0, 1.0, 0.3], p),
    "pressed": lambda p: p * [1.0, 1.0, 0.5],
    "drawn out": lambda p: p * [3.0, 1.0, 1.0],
}


@pytest.mark.parametrize("pose", POSES)
def test_large_records_leave_the_tile_form(pose):
    """One tile, some of whose clusters are far from their volume: rounded to 23 bits of the
    largest, the records of all would move the points by other amounts than the lists' floats do.
    Taken from the lists, the moves (up to 0.03) differ by the order of a few FP32 operations, a
    relative 2^-24, which turns one rounding in 25 of positions around 0.5; twice that is let pass."""
    scene = H.scenes.make_scene(128, 3)
    pos = POSES[pose](scene["pos"] * 1.01).astype(np.float32)
    tile, (tiles, rows) = _one_iteration(pos, scene, 0)
    lists, _ = _one_iteration(pos, scene, 4)
    assert tiles == 1 and rows == 0
    assert np.mean(tile != lists) < 0.08


def test_small_records_take_the_tile_form():
    """Swollen by 1 %: the tile form runs (its roundings show) and is off by at most 2^-27 of the
    largest coordinate, which can turn the rounding of a position, one unit of 2^-23, either way."""
    scene = H.scenes.make_scene(128, 3)
    pos = (scene["pos"] * 1.01).astype(np.float32)
    tile, (tiles, rows) = _one_iteration(pos, scene, 0)
    lists, _ = _one_iteration(pos, scene, 4)
    assert tiles == 1 and rows == 0
    assert (tile != lists).any()
    assert np.abs(tile.astype(np.float64) - lists).max() <= (2.0 ** -23 + 2.0 ** -27) * np.abs(pos).max()


def _settled(solver, n, mode):
    """Positions after 24 substeps of a pinned scene in ``mode``, and the tuner's figures."""
    scen = H.scenes.plain_scene_scenario(n, 2, pins=50)
    scen.setup(solver)
    _fused(solver, mode)
    scen.advance(solver, 24)
    return solver.positions(), _tuning(solver)


def test_one_round_of_the_solve_has_no_other_forms(lib):
    """Below two rounds the forms 2 and 3 would be form 0 again: they are not tried."""
    _, t = _settled(lib, 2500, 2)
    assert t[1] == 1.0 and t[0] in (0.0, 1.0) and t[2] > 0.0 and t[3] > 0.0
    assert t[5] == 0.0 and t[6] == 0.0


def test_forms_agree_above_two_rounds(lib):
    """94,800 rows: two rounds of the solve, in all its forms, under the autotuner."""
    out, t = _settled(lib, 94800, 2)
    assert t[1] == 1.0 and (t[[2, 3, 5, 6]] > 0.0).all()
    ref, _ = _settled(lib, 94800, 0)
    assert H.max_err_over_diag(out, ref, H.scenes.bbox_diagonal(ref)) < H.TOL_1STEP


def test_session_above_two_rounds_equals_alone():
    """Alone, 40,000 rows take eight rows a warp in the distance kernel and one round of the
    solve; in an arena of 100,000 both take the larger forms.  Same bits."""
    serve = H.pkg.serve

    def session(k, n):
        s = serve.Session(k, 0.0, n, 99, 300 + k)
        s.admit(H.B200_SO)
        return s

    sizes = (40000, 60000)
    rows = sum(sizes)
    arena = H.pkg.bridge.Arena(H.B200_SO, rows, rows * 12, rows * 66, rows * 68)
    live = [session(k, n) for k, n in enumerate(sizes)]
    for s in live:
        s.slot = arena.admit(s.solver)
        assert s.slot is not None
        s.solver.close()
    for _ in range(2):
        arena.step(10, *serve._frame_arrays(live, 10))
        arena.sync()
        for s in live:
            s.scen.k += 10
    got = [arena.positions(s.slot, s.n) for s in live]
    arena.close()
    for k, n in enumerate(sizes):
        alone = session(k, n)
        for _ in range(2):
            alone.enqueue_frame()
        alone.solver.lib.xpbd_b200_sync()
        np.testing.assert_array_equal(got[k], alone.solver.positions())
        alone.close(keep_result=False)


@pytest.mark.parametrize("value", [np.nan, np.inf, 1e20, 50.0])
def test_a_position_gone_astray_against_the_oracle(value):
    """One Gaussian far off or not finite, in the middle of a tile: the others as the oracle has
    them, finite where it has them finite."""
    scene = H.scenes.make_scene(1500, 5)
    pos = (scene["pos"] * [1.1, 0.95, 1.0]).astype(np.float32)
    pos[700, 1] = value
    out = []
    for solver in (H.b200(), H.oracle()):
        H.scenes.Scenario(scene, [], iters=1, shape=False).setup(solver)
        solver.step()
        solver.reset()
        solver.set_positions(pos)
        solver.step()
        out.append(solver.positions())
        solver.destroy()
    got, ref = out
    np.testing.assert_array_equal(np.isfinite(got), np.isfinite(ref))
    near = np.isfinite(ref).all(1) & (np.abs(ref).max(1) < 10.0)
    assert near.sum() >= 1480
    assert H.max_err_over_diag(got[near], ref[near], H.scenes.bbox_diagonal(ref[near])) < H.TOL_1STEP
