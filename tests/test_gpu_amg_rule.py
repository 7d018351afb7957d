"""The multigrid's lanes per row follow from the hierarchy alone: fresh grids
of one specimen get the same lanes, and so, as a row's sum is formed in the
order that its lanes give, the same potentials to the bit and the same events."""
import numpy as np
import pytest

from conftest import SMALL_TIP

pytestmark = pytest.mark.gpu

# about 85k cells: a first coarse level of 6,500 rows, where timed lanes
# differed most from grid to grid
MIDDLE = dict(SMALL_TIP, cap_radius=3.2e-9, shank_length=6e-9, box_half_width=0.5e-6, box_height=1.0e-6,
              fine_shell=2.2e-9)


@pytest.mark.parametrize("tip", [SMALL_TIP, MIDDLE], ids=["small", "middle"])
def test_fresh_grids_agree_to_the_bit(tip):
    from tapsim_modified_b200.tapsim import Evaporation, EvaporationOptions, Grid, Mesh, solve_opts
    mesh = Mesh.from_tip(**tip)
    lanes, phi, voltages = [], [], []
    for _ in range(6):
        g = Grid(mesh)
        g.surface_init(0)
        g.solve(1e-10, 50, 50000, 1e-4, preconditioner=1)
        lanes.append([(lv["a_lanes"] if lv["level"] else 0, lv["r_lanes"]) for lv in g.amg_schedule()])
        phi.append(g.potentials())
        ev = Evaporation(g, EvaporationOptions.from_ini(None), relax_mode=1,
                         solve=solve_opts(rel_tol=1e-8, max_outer=50, max_inner=20000, preconditioner=1))
        voltages.append([r["voltage"] for r in ev.run(2)])
        g.close()
    assert len(phi[0]) > (60000 if tip is MIDDLE else 0)
    assert all(x == lanes[0] for x in lanes), lanes
    assert all(np.array_equal(p, phi[0]) for p in phi)
    assert all(v == voltages[0] for v in voltages), voltages
