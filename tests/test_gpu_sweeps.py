"""Coloured sweeps (Grid.relax) against the same sweeps in numpy: greedy
colours in index order over the whole neighbour graph, the rows of a colour
updated together, n sweeps; rows with fewer and with more couplings than a
thread loads ahead (16), non-Neumann and Neumann rows in one launch."""
import numpy as np
import pytest

from conftest import SMALL_TIP

pytestmark = pytest.mark.gpu


def _sweeps(a, n):
    rp, col = a["row_ptr"], a["col"]
    N = len(a["type"])
    colour = np.full(N, -1)
    for i in range(N):
        used = set(colour[col[rp[i]:rp[i + 1]]].tolist())
        c = 0
        while c in used:
            c += 1
        colour[i] = c
    types = a["types"]
    neumann = np.isin(a["type"], [t for t, v in types.items() if v["neumann"]])
    free = ~np.isin(a["type"], [t for t, v in types.items() if v["dirichlet"]])
    row = np.repeat(np.arange(N), np.diff(rp))
    c64 = np.where(~neumann[row] & neumann[col], 0.0, a["coupling"])
    phi = a["phi"].astype(np.float64)
    entries = [np.nonzero(free[row] & (colour[row] == c))[0] for c in range(colour.max() + 1)]
    for _ in range(n):
        dev = 0.0
        for e in entries:
            rows = np.unique(row[e])
            if not len(rows):
                continue
            s = np.bincount(row[e], weights=c64[e] * phi[col[e]], minlength=N)[rows]
            d = np.bincount(row[e], weights=c64[e], minlength=N)[rows]
            dev = max(dev, np.abs(s / d - phi[rows]).max())
            phi[rows] = s / d
    return phi, dev


@pytest.mark.parametrize("n", [1, 2, 7])
@pytest.mark.parametrize("spacing", [0.0, 1.2e-9])
def test_sweeps_match_numpy(n, spacing):
    from tapsim_modified_b200.tapsim import Grid, Mesh
    mesh = Mesh.from_tip(**dict(SMALL_TIP, max_spacing=spacing))
    a = mesh.arrays()
    lengths = np.diff(a["row_ptr"])
    assert lengths.min() < 16 < lengths.max()
    g = Grid(mesh)
    dev = g.relax(n)
    phi, ref = _sweeps(a, n)
    # sums of at most some tens of terms of one sign, n sweeps of averaging
    assert np.abs(g.potentials() - phi).max() <= 1e-13
    assert abs(dev - ref) <= 1e-13
