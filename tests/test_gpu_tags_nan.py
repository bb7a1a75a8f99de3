"""The interface criterion beside a volume fraction that is not a number.  With two solids the larger
fraction decides, and the second where the first is no number (the reference's comparison a0 > a1
selects it); such a cell still shows a crossing to its neighbours."""
import numpy as np
import pytest

from forestfv_public_gb300 import Mesh, Solver, uniform_leaves
from forestfv_public_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("second,crossing", [(0.9, True), (0.1, False)])
def test_first_solid_fraction_not_a_number(second, crossing, built_lib):
    mesh = Mesh((1, 1, 1), uniform_leaves((1, 1, 1), 4))
    m, n = W.WALL, mesh.n
    S = W.wall_state(m, np.zeros(n, bool), np.full(n, 0.5))
    S[7], S[8] = 0.2, 0.3
    x = mesh.centroids() / mesh.centroids().max()
    c = int(np.argmin(np.abs(x - 0.5).sum(axis=1)))
    S[7, c], S[8, c] = np.nan, second
    s = Solver(model=5, gamma=m["gamma"], pinf=m["pinf"], mu=[2.6e10, 1e10, 0.0], amin=m["amin"], avf_lim=0.5,
               prelax=3)
    s.set_mesh(mesh)
    s.upload_state(S)
    _, _, si = s.tags((0, 4, 0, 0, 0.0, 0, 0, 0.0, 0, 0, 0.0, 1, 5, 2, 0, 0, 0), with_raw=True)
    s.close()
    h = np.diff(np.unique(x[:, 0])).min()
    near = np.abs(x - x[c]).sum(axis=1) < 1.5 * h  # the cell and its six neighbours
    assert near.sum() == 7
    assert np.array_equal(si[0] == 1, near if crossing else np.zeros(n, bool))
