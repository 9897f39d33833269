"""ChainMail waves that leave most of the scene alone: sweeps skip what they do not reach."""
import numpy as np
import pytest

import helpers as H

pytestmark = pytest.mark.gpu


def _scene(n, hubs):
    """The plain graph plus ``hubs`` Gaussians joined to every third other one, with rest lengths
    1 % off: at rest, whether an edge pulls is a matter of rounding."""
    sc = H.scenes.make_scene(n, 3)
    more = np.concatenate([np.zeros((0, 2), np.int64)] +
                          [np.stack([np.full(len(range(1, n, 3)), h), np.arange(1, n, 3)], 1) for h in hubs])
    edges = np.unique(np.sort(np.concatenate([sc["edges"], more[more[:, 0] != more[:, 1]]]), axis=1), axis=0)
    d = sc["pos"][edges[:, 0]].astype(np.float64) - sc["pos"][edges[:, 1]]
    sc["edges"] = edges.astype(np.int32)
    sc["rest"] = (1.01 * np.sqrt((d * d).sum(1))).astype(np.float32)
    sc["stiff"] = np.where(np.arange(len(edges)) % 3 == 0, 0.5, 1.0).astype(np.float32)
    return sc


# blocks of 1,024 rows: one, a remainder of one row, several; rows whose edges lead to more blocks
# than a warp lists (hubs, 12 blocks); waves that are under way, and long over, when the run ends
@pytest.mark.parametrize("n,hubs,sweeps", [(1024, (), 5), (1025, (), 6), (6000, (), 4), (6000, (), 90),
                                           (12000, (0, 7000), 3), (12000, (11999,), 40)])
def test_waves_equal_dense_sweeps_and_oracle(n, hubs, sweeps):
    """Two pushes, the second while the first wave is still a flag of changed rows.  Arrival times
    are sums and minima of the same constants in the same order: equal.  Positions equal those of
    sweeps over every Gaussian, and after the first run the oracle's; its closing relax sweep leaves
    edges at their rest length, where the second one's count of pulling edges is a matter of
    rounding."""
    sc = _scene(n, hubs)
    far = np.argsort(sc["pos"][:, 0])
    out = []
    for solver, frontier in ((H.b200(), 1), (H.b200(), 0), (H.oracle(), None)):
        H.scenes.Scenario(sc, [], iters=1, ring_k=1, max_members=8).setup(solver)
        solver.step()
        solver.reset()
        if frontier is not None:
            solver.lib.xpbd_b200_chainmail_set_frontier(frontier)
        runs = []
        for k, seeds in enumerate((far[:3], far[-3:])):
            solver.chainmail_seed(seeds.astype(np.int32), np.full((3, 3), 0.01 * (1 - 2 * k), np.float32))
            solver.chainmail_run(**{**H.scenes.CHAINMAIL_DEFAULTS, "prop_iters": sweeps + k, "relax_iters": 0})
            runs.append((solver.positions(), solver.chainmail_times()))
        out.append(runs)
        if frontier is not None:
            solver.lib.xpbd_b200_chainmail_set_frontier(1)
        solver.destroy()
    for (p, t), (p_all, t_all), (_, u) in zip(*out):
        np.testing.assert_array_equal(p, p_all)
        np.testing.assert_array_equal(t, t_all)
        np.testing.assert_array_equal(t, u)
    p, q = out[0][0][0], out[2][0][0]
    assert H.max_err_over_diag(p, q, H.scenes.bbox_diagonal(q)) < H.TOL_1STEP
