"""tg_solve's cap of inner iterations at the bottom of its range: below 0 it
is refused before anything runs; at 0 a fresh handle's solve keeps to its
cap of outer steps and leaves a state that an ordinary solve converges from."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cap", [-1, -3])
def test_negative_cap_is_refused(small_mesh, cap):
    from tapsim_modified_b200 import _native as N
    from tapsim_modified_b200.tapsim import Grid
    g = Grid(small_mesh)
    before = g.potentials()
    with pytest.raises(N.TapsimError) as e:
        g.solve(rel_tol=1e-8, max_outer=2, max_inner=cap, preconditioner=1)
    assert e.value.code == N.TG_ERR_ARGUMENT
    assert np.array_equal(g.potentials(), before)
    g.close()


@pytest.mark.parametrize("mode", [0, 1, 2])
def test_cap_of_zero(small_mesh, mode):
    from tapsim_modified_b200 import _native as N
    from tapsim_modified_b200.tapsim import Grid
    g, other = Grid(small_mesh), Grid(small_mesh)
    g.set_launch_mode(mode)
    with pytest.raises(N.TapsimError) as e:
        g.solve(rel_tol=1e-10, max_outer=2, max_inner=0, preconditioner=1)
    assert e.value.code == N.TG_ERR_ITERATION_CAP
    for x in (g, other):
        assert x.solve(rel_tol=1e-11, max_outer=50, max_inner=20000, preconditioner=1).rel_residual <= 1e-11
    # two solutions to 1e-11 of ||b||, potentials up to 1 (as the solves of
    # different starts are compared elsewhere)
    assert np.abs(g.potentials() - other.potentials()).max() <= 1e-8
    g.close()
    other.close()
