"""The deformed-shape writeback, bit for bit.

Where two axes are nearly equal the last bit of Sigma decides their order and signs, which a
caller that compares or interpolates scales and rotations sees, so the roundings of the
eigen-decompositions are part of the result.  tests/golden/shapes_bits.npz holds the scales
and rotations that the library returned on a B200 when the 3x3 matrices were indexed in local
memory."""
import numpy as np
import pytest

import helpers as H

pytestmark = pytest.mark.gpu


def writeback(solver):
    """Shapes of the 4,000-Gaussian scene at its recorded positions after 100 steps; every
    other Gaussian a ball, whose axes the deformation alone decides."""
    g = H.load_golden("plain_n4000")
    scene = H.golden_scene(g)
    scene["scales"][::2] = 0.02
    H.scenes.Scenario(scene, []).setup(solver)
    solver.step()
    solver.reset()
    solver.set_positions(g["pos_100"])
    return solver.shapes(1e-4)


def test_writeback_keeps_its_bits():
    gold = H.load_golden("shapes_bits")
    lib = H.b200()
    scales, rotations, deformed = writeback(lib)
    lib.destroy()
    assert deformed == int(gold["deformed"]) > 3000
    np.testing.assert_array_equal(scales[gold["rows"]], gold["scales"])
    np.testing.assert_array_equal(rotations[gold["rows"]], gold["rotations"])
