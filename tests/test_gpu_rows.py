"""Distance and shape matching on rows and rotations at their limits, against the oracle."""
import numpy as np
import pytest

import helpers as H

pytestmark = pytest.mark.gpu


def _rotated(p):
    a, k = 3.0, np.array([0.6, 0.0, 0.8])
    c, s = np.cos(a), np.sin(a)
    return c * p + s * np.cross(k, p) + (1 - c) * (p @ k)[:, None] * k


POSES = {
    "rest": lambda p: p,
    "turned": _rotated,                                  # 172 degrees from the last rotation
    "flat": lambda p: p * np.array([1.0, 1.0, 1e-3]),    # one singular value near zero
    "mirrored": lambda p: p * np.array([-1.0, 1.0, 1.0]),
}


def _hub_scene(n, hubs):
    """The plain graph plus ``hubs`` Gaussians joined to every other one: rows longer than the
    kernels' shared-memory windows."""
    sc = H.scenes.make_scene(n, 3)
    key = sc["edges"][:, 0].astype(np.int64) * n + sc["edges"][:, 1]
    more = np.concatenate([key[:0]] + [np.minimum(h, np.arange(n)) * np.int64(n) + np.maximum(h, np.arange(n))
                                       for h in hubs])
    key = np.unique(np.concatenate([key, more[more // n != more % n]]))
    sc["edges"] = np.stack([key // n, key % n], 1).astype(np.int32)
    d = sc["pos"][sc["edges"][:, 0]].astype(np.float64) - sc["pos"][sc["edges"][:, 1]]
    sc["rest"] = np.sqrt((d * d).sum(1)).astype(np.float32)
    sc["stiff"] = np.where(np.arange(len(key)) % 3 == 0, 0.5, 1.0).astype(np.float32)
    return sc


@pytest.mark.parametrize("n,hubs,pose,robust", [
    (31, (), "rest", True), (33, (), "turned", True), (1000, (), "turned", True), (1000, (), "flat", True),
    (1000, (), "mirrored", True), (1000, (), "turned", False), (700, (0, 350), "rest", True),
    (2000, (5, 6, 1999), "turned", True)])
def test_rows_and_rotations_match_oracle(n, hubs, pose, robust):
    """One substep of two iterations, distance and shape matching; the one-step tolerance."""
    sc = _hub_scene(n, hubs)
    pos = POSES[pose](sc["pos"].astype(np.float64)) * 1.02
    out = []
    for solver in (H.b200(), H.oracle()):
        scen = H.scenes.Scenario(sc, [], iters=2, volume=False, shape_robust=robust)
        scen.setup(solver)
        solver.step()
        solver.reset()
        solver.set_positions(pos.astype(np.float32))
        solver.step()
        out.append(solver.positions())
        solver.destroy()
    assert np.isfinite(out[1]).all()
    assert H.max_err_over_diag(out[0], out[1], H.scenes.bbox_diagonal(out[1])) < H.TOL_1STEP


@pytest.mark.parametrize("n", [9, 42624, 42625])
def test_rows_per_warp_match_oracle(n):
    """Distance on both sides of the limit where a warp takes 8 rows instead of 32 (148 SMs x 9
    blocks x 4 warps x 8 rows); the one-step tolerance."""
    sc = _hub_scene(n, (0,) if n > 1000 else ())
    out = []
    for solver in (H.b200(), H.oracle()):
        scen = H.scenes.Scenario(sc, [], iters=2, volume=False, shape=False)
        scen.setup(solver)
        solver.step()
        out.append(solver.positions())
        solver.destroy()
    assert H.max_err_over_diag(out[0], out[1], H.scenes.bbox_diagonal(out[1])) < H.TOL_1STEP
