"""ChainMail sweeps on rows and sweep counts at their limits, against the oracle."""
import numpy as np
import pytest

import helpers as H
from test_gpu_rows import _hub_scene

pytestmark = pytest.mark.gpu


# 31, 32, 33: around a mask word; 1000 with hubs: rows longer than the kernels' windows; odd and
# even sweep counts: which copy of the state a run ends on; 40 sweeps of 300: past the last change
@pytest.mark.parametrize("frontier", [1, 0])
@pytest.mark.parametrize("n,hubs,sweeps", [(31, (), 3), (32, (), 2), (33, (), 1), (300, (), 40), (1000, (0, 500), 3)])
def test_sweeps_match_oracle(n, hubs, sweeps, frontier):
    """Repeated seeds, then two runs of propagation and one relax sweep: arrival times are sums
    and minima of a few constants taken in the same order, so they are equal; positions to the
    one-step tolerance."""
    sc = _hub_scene(n, hubs)
    # off the rest pose: the relax sweep divides by the number of edges more than about 1e-7 from
    # their rest length, which for edges at rest is a matter of rounding
    sc["rest"] = (sc["rest"] * np.float32(1.01)).astype(np.float32)
    seeds = np.array([0, 5, n - 1, 5, 0, 0], np.int32)
    push = np.full((len(seeds), 3), 0.02, np.float32) * np.arange(1, 7, dtype=np.float32)[:, None]
    out = []
    for solver in (H.b200(), H.oracle()):
        scen = H.scenes.Scenario(sc, [], iters=1)
        scen.setup(solver)
        solver.step()      # uploads the graph
        solver.reset()
        if solver.prefix == "b200":
            solver.lib.xpbd_b200_chainmail_set_frontier(frontier)
        for k in range(2):
            solver.chainmail_seed(seeds, push * (1 - 2 * k))
            solver.chainmail_run(**{**H.scenes.CHAINMAIL_DEFAULTS, "prop_iters": sweeps + k, "relax_iters": 0})
        out.append((solver.positions(), solver.chainmail_times()))
        if solver.prefix == "b200":
            solver.lib.xpbd_b200_chainmail_set_frontier(1)
        solver.destroy()
    (p, t), (q, u) = out
    assert np.isfinite(q).all() and (u[seeds] == 0).all()
    np.testing.assert_array_equal(t, u)
    assert H.max_err_over_diag(p, q, H.scenes.bbox_diagonal(q)) < H.TOL_1STEP
