"""Edges of the inner solve's one-launch forms against its kernels launched
one by one (mode 0): Neumann rows with more neighbours of their kind than the
cluster kernel keeps in shared memory (12), and the captured solve's slots as
removals cross a multiple of 1024 and reach the end of the append reserve."""
import numpy as np
import pytest

from conftest import SMALL_TIP

pytestmark = pytest.mark.gpu

SOLVE = dict(rel_tol=1e-10, max_outer=50, max_inner=20000, preconditioner=1)


def _neumann(a):
    return np.isin(a["type"], [t for t, v in a["types"].items() if v["neumann"]])


@pytest.mark.parametrize("spacing, x_min", [(0.0, 2e-9), (0.7e-9, 7e-9)])
def test_wide_neumann_rows(tmp_path, spacing, x_min):
    from tapsim_modified_b200.tapsim import Grid, Mesh
    m = Mesh.from_tip(**dict(SMALL_TIP, max_spacing=spacing))
    a = m.arrays()
    side = next(t for t, v in a["types"].items() if v["neumann"] and np.any(a["type"] == t))
    m.write_node_file(str(tmp_path / "t.nodes"))
    m.write_config(str(tmp_path / "t.cfg"))
    # the vacuum cells of one side of the box become Neumann cells
    head, body = (tmp_path / "t.nodes").read_bytes().split(b"\n", 1)
    rec = np.frombuffer(body, dtype=[("xyz", "<f4", 3), ("id", "<i2")]).copy()
    rec["id"][(rec["id"] == 0) & (rec["xyz"][:, 0] > x_min)] = side
    (tmp_path / "w.nodes").write_bytes(head + b"\n" + rec.tobytes())
    mesh = Mesh.from_files(str(tmp_path / "w.nodes"), str(tmp_path / "t.cfg"))
    a = mesh.arrays()
    neumann = _neumann(a)
    row = np.repeat(np.arange(len(neumann)), np.diff(a["row_ptr"]))
    kind = np.bincount(row, weights=neumann[row] & neumann[a["col"]], minlength=len(neumann))
    assert kind.max() > 12 and neumann.sum() <= 16384
    out = {}
    for mode in (0, 2):
        g = Grid(mesh)
        g.set_launch_mode(mode)
        info = g.solve(**SOLVE)
        assert info.rel_residual <= 1e-10 and g.residual() <= 1e-10 and info.inner_neumann > 0
        out[mode] = (info.inner_neumann, g.potentials())
        g.close()
    # the same iterations up to the order of the double sums
    assert abs(out[0][0] - out[2][0]) <= max(2, 0.1 * out[0][0])
    assert np.abs(out[0][1] - out[2][1]).max() <= 1e-8


@pytest.mark.parametrize("removals", [31, 33, 1060])
def test_slots_across_a_boundary_and_at_the_reserve(removals):
    """The V rows' slots end 32 before a multiple of 1024; the reserve ends
    less than 1024 past the next one, which 1,057 removals pass."""
    from tapsim_modified_b200.tapsim import Grid, Mesh
    mesh = Mesh.from_tip(**dict(SMALL_TIP, fine_shell=5.85e-10))
    a = mesh.arrays()
    types = a["types"]
    free = ~np.isin(a["type"], [t for t, v in types.items() if v["dirichlet"]])
    slots = (int((free & ~_neumann(a)).sum()) + 31) // 32 * 32
    reserve = (int(np.isin(a["type"], [t for t, v in types.items() if v["removable"]]).sum()) + 31) // 32 * 32
    assert slots % 1024 == 992 and 1024 < reserve < 2048 and (slots + reserve) % 1024
    out = {}
    for mode in (0, 2):
        g = Grid(mesh)
        g.set_launch_mode(mode)
        g.surface_init(0)
        g.solve(**SOLVE)
        gone = 0
        while gone < removals:
            for node in sorted(g.surface()[0].tolist()):
                if gone < removals and g.types()[node] != 0:
                    gone += 1 + len(g.take_away(node))
        info = g.solve(**SOLVE)
        assert info.rel_residual <= 1e-10 and g.residual() <= 1e-10
        out[mode] = (gone, g.types(), g.potentials())
        g.close()
    assert out[0][0] == out[2][0] and np.array_equal(out[0][1], out[2][1])
    assert np.abs(out[0][2] - out[2][2]).max() <= 1e-8
