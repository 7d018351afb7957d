"""Training calls of more steps than are staged at a time (64): the losses of
the steps on both sides of the boundary against the same steps taken one call
each, on one sample (every batch is then the same, whatever the draw)."""
import numpy as np
import pytest

from conftest import GOLDEN

pytestmark = pytest.mark.gpu


def _learner(mesh):
    from tapsim_modified_b200.tapsim import EvaporationOptions, Evaporation, Grid, Learner, solve_opts
    g = Grid(mesh)
    g.solve(rel_tol=1e-10)
    L = Learner(hops=4, max_cells=4096, ell_width=64, seed=3)
    L.attach(g, collect=True)
    Evaporation(g, EvaporationOptions.from_ini(str(GOLDEN / "oracle.ini")), relax_mode=1,
                solve=solve_opts(rel_tol=1e-10, warm_start=1, preconditioner=1)).run(3)
    L.attach(g)
    return L


@pytest.mark.parametrize("batch", [1, 3])
def test_steps_across_the_staged_ones(ref_mesh, batch):
    a, b = _learner(ref_mesh), _learner(ref_mesh)
    kw = dict(batch=batch, lr=1e-4, first=1, count=1)
    first = a.gradients(1, 1)[0]
    # 70 steps: mean_loss is the mean of the last seven, steps 63..69
    together = a.train(70, **kw)
    b.train(63, **kw)
    apart = np.mean([b.train(1, **kw) for _ in range(7)])
    assert np.isfinite(together) and together < first
    # Adam moves a parameter by at most about lr a step, also one whose
    # gradient is rounding noise: after 63 steps the two trainings' losses
    # agree to a few per cent, while another row's sample or an empty batch
    # would not
    assert abs(together - apart) <= 0.05 * apart
    # and the steps went on from one another: the next loss is below the mean
    assert a.gradients(1, 1)[0] <= 1.05 * together
    assert a.train(0, **kw) == 0.0
