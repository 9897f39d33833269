"""Shape matching's rotation, found from the one before, at poses where that one misleads."""
import numpy as np
import pytest

import helpers as H

pytestmark = pytest.mark.gpu


def _stars(stretch):
    """27 Gaussians with six neighbours each, an octahedron with arms 0.1 * stretch about a point
    0.01 away: neighbourhoods that look nearly the same along every axis."""
    rng = np.random.default_rng(4)
    at = 0.5 * (np.stack(np.meshgrid(*[np.arange(3)] * 3, indexing="ij"), -1).reshape(-1, 3) - 1.0)
    off = rng.standard_normal((27, 3))
    off *= 0.01 / np.linalg.norm(off, axis=1, keepdims=True)
    arms = 0.1 * np.concatenate([np.diag(stretch), -np.diag(stretch)])
    pos = np.concatenate([(at + off)[:, None], at[:, None] + arms], 1).reshape(-1, 3).astype(np.float32)
    edges = np.stack([np.repeat(np.arange(27) * 7, 6), np.arange(27 * 7).reshape(27, 7)[:, 1:].ravel()], 1)
    d = pos[edges[:, 0]].astype(np.float64) - pos[edges[:, 1]]
    n = len(pos)
    return {"pos": pos, "scales": np.full((n, 3), 0.02, np.float32),
            "rots": np.tile(np.float32([1, 0, 0, 0]), (n, 1)), "opacity": np.full(n, 0.9, np.float32),
            "edges": edges.astype(np.int32), "rest": np.sqrt((d * d).sum(1)).astype(np.float32),
            "stiff": np.ones(len(edges), np.float32)}


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("stretch", [0.004, 0.0])
def test_half_turn_of_an_isotropic_neighbourhood(axis, stretch):
    """The rest pose, half a turn about the axis it is stretched along: shape matching leaves it
    where it is, whatever the rotation before."""
    scene = _stars(1.0 + stretch * np.eye(3)[axis])
    turned = scene["pos"] * np.where(np.arange(3) == axis, 1.0, -1.0).astype(np.float32)
    got = []
    for solver in (H.b200(), H.oracle()):
        H.scenes.Scenario(scene, [], volume=False).setup(solver)
        solver.step()
        solver.reset()
        solver.set_positions(turned)
        solver.step()
        got.append(solver.positions())
        solver.destroy()
    diag = H.scenes.bbox_diagonal(turned)
    assert H.max_err_over_diag(got[0], got[1], diag) < H.TOL_1STEP
    assert H.max_err_over_diag(got[0], turned, diag) < H.TOL_1STEP
