"""Tile ranges and their order for short pair lists, single tiles and wide keys, against the
oracle."""
import numpy as np
import pytest

import helpers
from test_render import Camera, assert_frames_close, pkg

pytestmark = pytest.mark.gpu


# 16x16: one tile; 33 Gaussians in 160x120: lists that end inside a 16-byte load; 4112x4112: 66,049
# tiles, whose keys take four bytes, nearly all of them empty
@pytest.mark.parametrize("n,W,H", [(1, 16, 16), (33, 16, 16), (33, 160, 120), (2000, 40, 24), (7, 4112, 4112)])
def test_bins_match_oracle(n, W, H):
    sc = pkg.scenes.make_scene(n, 5)
    if W > 4096:
        sc["scales"] = (sc["scales"] * np.float32(0.05)).astype(np.float32)   # a few tiles each
    solver = pkg.bridge.XPBD(helpers.B200_SO)
    try:
        scen = pkg.scenes.Scenario(sc, [], iters=1)
        scen.setup(solver)
        solver.step()
        pos = solver.positions()
        colors = pkg.splat.synthetic_colors(n, -1, 2)
        solver.render_set_colors(colors)
        solver.render_set_options()
        solver.render_set_floor(False)
        cam = Camera.framing(np.concatenate([pos, pos + 0.1]), W, H)
        img, m = solver.render(cam, deform_eps=-1.0, bg=(0.1, 0.2, 0.3))
        ft, nc, _, radii = solver.render_aux(W, H)
    finally:
        solver.destroy()
    ref = helpers.oracle_render(pos, sc["scales"], sc["rots"], sc["opacity"], colors, -1, cam, bg=(0.1, 0.2, 0.3))
    assert ref["pairs"] > 0
    assert_frames_close({"image": img, "final_T": ft, "n_contrib": nc, "radii": radii, "pairs": m}, ref, f"{n} {W}x{H}")
