"""All-FP32 flights whose positions stay on a mesh vertex for many trials (a
step there is below a float's spacing): a retried trial starts its walks from
the state's tetrahedron, whatever tetrahedra the rejected trial's stages ended
in, so that the tetrahedra of such a vertex are taken in one order.  The
potentials are zero inside a cylinder and rise outside, so that on its edge
the interpolated fields differ between a vertex's tetrahedra in more than
their last digits; the expected trials are those of one thread per ion that
walks to every point."""
import numpy as np
import pytest

from conftest import QM_FE, SMALL_TIP

pytestmark = pytest.mark.gpu

# trials by index in the sorted surface set
TRIALS = {216: 735, 278: 694, 283: 646, 286: 655, 406: 700, 498: 663, 502: 715, 507: 691, 537: 716, 543: 723}


def test_retried_trials_start_from_the_states_tetrahedron(small_mesh):
    from tapsim_modified_b200.tapsim import Grid
    a = small_mesh.arrays()
    g = Grid(small_mesh)
    g.surface_init(0)
    x = a["xyz"].astype(np.float64)
    g.set_potentials(-3000.0 * np.maximum(np.hypot(x[:, 0], x[:, 1]) - SMALL_TIP["cap_radius"], 0) / x[:, 2].max())
    nodes = np.sort(g.surface()[0])
    imp = np.ctypeslib.as_array(g.trace(a["xyz"][nodes], QM_FE, a["node_tet"][nodes], precision=1, max_steps=400))
    assert {k: int(imp["trials"][k]) for k in TRIALS} == TRIALS
    g.close()
