"""The Neumann rows' inner solve in one launch of a cluster (launch modes 1
and 2) against its kernels launched one by one (mode 0), at row counts on
both sides of one, two, three and four rows per thread (4096 each) and past
the limit, where mode 2 takes the kernels too."""
import numpy as np
import pytest

from conftest import SMALL_TIP

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spacing, per_thread", [(0.0, 1), (1.2e-9, 1), (0.9e-9, 2), (0.7e-9, 2), (0.6e-9, 3),
                                                 (0.5e-9, 4), (0.45e-9, 5)])
@pytest.mark.parametrize("precision", [0, 1])
def test_one_launch_matches_the_kernels(spacing, per_thread, precision):
    from tapsim_modified_b200.tapsim import Grid, Mesh
    if precision and per_thread > 2:
        pytest.skip("the FP64 inner correction reaches the rows the same way at any count")
    mesh = Mesh.from_tip(**dict(SMALL_TIP, max_spacing=spacing))
    a = mesh.arrays()
    rows = int(np.isin(a["type"], [t for t, v in a["types"].items() if v["neumann"]]).sum())
    assert (rows + 4095) // 4096 == per_thread
    out = {}
    for mode in (0, 2):
        g = Grid(mesh)
        g.set_launch_mode(mode)
        info = g.solve(rel_tol=1e-10, max_outer=50, max_inner=20000, preconditioner=1, inner_precision=precision)
        out[mode] = (info.inner_neumann, g.potentials())
        assert info.rel_residual <= 1e-10 and g.residual() <= 1e-10
        g.close()
    # the same iterations up to the order of the double sums
    assert abs(out[0][0] - out[2][0]) <= max(2, 0.1 * out[0][0])
    assert np.abs(out[0][1] - out[2][1]).max() <= 1e-8
