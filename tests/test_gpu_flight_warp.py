"""Flights by one warp per ion: points found among the warp's tetrahedra
against points found by walking alone.

With a walk bound below 256 every point is located by a walk from the last
one's tetrahedron; above, by the tetrahedra the warp holds where one of them
holds the point.  The tetrahedron found is the same unless the point lies on
a shared face to rounding, so nearly every flight is the same to the bit, and
the rest stay within the bound that separate flights keep to the oracle."""
import numpy as np
import pytest

from conftest import QM_FE

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def grid(small_mesh):
    from tapsim_modified_b200.tapsim import Grid
    g = Grid(small_mesh)
    g.solve(rel_tol=1e-10)
    g.surface_init(0)
    return g, small_mesh.arrays()


@pytest.mark.parametrize("precision", [0, 1, 2])
@pytest.mark.parametrize("ions", [1, 33, 1300])
def test_located_and_walked_flights_agree(grid, ions, precision):
    g, a = grid
    nodes, _ = g.surface()
    pick = np.random.default_rng(5).choice(nodes, ions, replace=ions > len(nodes))
    kw = dict(precision=precision, fp64_radius=5e-9)
    hit = np.ctypeslib.as_array(g.trace(a["xyz"][pick], QM_FE, a["node_tet"][pick], **kw))
    walked = np.ctypeslib.as_array(g.trace(a["xyz"][pick], QM_FE, a["node_tet"][pick], walk_limit=255, **kw))
    assert np.all(hit["status"] == 5) and np.all(walked["status"] == 5)
    same = (hit["trials"] == walked["trials"]) & np.all(hit["stop"] == walked["stop"], axis=1)
    assert np.mean(same) >= 0.95
    d = np.hypot(*(hit["stop"] - walked["stop"])[:, :2].T) / np.hypot(*walked["stop"][:, :2].T)
    assert d.max() <= 2e-2
