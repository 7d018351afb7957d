"""Batches of the learned start's training: the batch gathered by one kernel,
its weight gradients from K chunks shared out over CTAs, whatever its rows'
remainder."""
import numpy as np
import pytest

from conftest import GOLDEN

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def learner(ref_mesh):
    from tapsim_modified_b200.tapsim import EvaporationOptions, Evaporation, Grid, Learner, solve_opts
    g = Grid(ref_mesh)
    g.solve(rel_tol=1e-10)
    L = Learner(hops=6, max_cells=4096, ell_width=64, seed=3)
    L.attach(g, collect=True)
    Evaporation(g, EvaporationOptions.from_ini(str(GOLDEN / "oracle.ini")), relax_mode=1,
                solve=solve_opts(rel_tol=1e-10, warm_start=1, preconditioner=1)).run(6)
    L.attach(g)
    return L


@pytest.mark.parametrize("count", [2, 3, 5])
def test_batch_gradient_is_the_mean_of_its_samples(learner, count):
    """A batch's loss and gradient are its samples' means weighted by their
    rows; the BF16 rounding of the gradients on the way (2^-9 relative, each
    value) differs with the batch's scale."""
    rows = np.array([learner.sample(k)["target"].size for k in range(count)])
    single = [learner.gradients(k, 1) for k in range(count)]
    loss, grad, out = learner.gradients(0, count)
    w = rows / rows.sum()
    assert abs(loss - sum(a * s[0] for a, s in zip(w, single))) <= 1e-5 * abs(loss)
    mean = sum(a * s[1].astype(np.float64) for a, s in zip(w, single))
    assert np.linalg.norm(grad - mean) <= 1e-2 * np.linalg.norm(mean)
    # a row's output does not depend on the batch
    assert np.abs(out - np.concatenate([s[2] for s in single])).max() <= 1e-5 * np.abs(out).max()
