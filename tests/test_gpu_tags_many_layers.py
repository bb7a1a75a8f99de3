"""More interface layers than 16 bits hold: a bar of 2 x 2 x 70,000 cells whose solid fraction crosses
AVF_LIM at one end, asked for layers up to the other.  A cell k steps from the interface is in layer
k.  Identical layers and levels, before and after calls with few layers on the same context."""
import numpy as np
import pytest

from forestfv_public_gb300 import Mesh, Solver, uniform_leaves
from forestfv_public_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def test_layers_beyond_16_bits(built_lib):
    mesh = Mesh((1, 1, 35000), uniform_leaves((1, 1, 35000), 2))
    m, n = W.WALL, mesh.n
    k = np.rint(mesh.centroids()[:, 2] / (0.5 * mesh.tree_edge) - 0.5).astype(np.int64)
    assert k.min() == 0 and k.max() == 69999
    S = W.wall_state(m, k < 1, np.zeros(n))
    s = Solver(model=5, gamma=m["gamma"], pinf=m["pinf"], mu=m["mu"], amin=m["amin"], avf_lim=0.5, prelax=3)
    s.set_mesh(mesh)
    s.upload_state(S)
    for layers in (20, 66000, 90000, 20):
        p = (0, 2, 0, 0, 0.0, 0, 0, 0.0, 0, 0, 0.0, 1, 3, layers, 0, 0, 0)
        _, raw, si = s.tags(p, with_raw=True)
        want = np.where(np.maximum(k, 1) < layers, np.maximum(k, 1), 0)
        for v in range(2):  # the solid's and the liquid's fraction cross together
            assert np.array_equal(si[v], want), (layers, v, int((si[v] != want).sum()))
        assert np.array_equal(raw, np.where((want > 0) & (want < layers), 3, 1)), layers
    s.close()
