"""A new mesh that fits the context's buffers allocates nothing on the device, however many of its faces
are boundary, coarser or finer ones: a strip of single-cell trees, one thick and three wide
(2.7 boundary faces a cell), after a cube of more cells; and a step on it gives the bits of a context that held nothing else."""
import numpy as np
import pytest
import torch

from forestfv_public_gb300 import Mesh, Solver, uniform_leaves
from forestfv_public_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def test_strip_after_cube(built_lib):
    m = W.WALL
    args = dict(model=5, gamma=m["gamma"], pinf=m["pinf"], mu=m["mu"], amin=m["amin"], avf_lim=0.5, prelax=3,
                flux_form=1, precision=1)
    cube = Mesh((2, 2, 2), uniform_leaves((2, 2, 2), 6))
    strip = Mesh((3, 1, 65536), uniform_leaves((3, 1, 65536), 1), tree_edge=0.5)
    n = strip.n
    assert 1.25 * cube.n + 1024 < 2.5 * n and n < cube.n
    z = strip.centroids()[:, 2]
    S = W.wall_state(m, z < 0.4 * z.max(), 0.5 + 0.4 * np.sin(z))
    out = []
    s = Solver(**args)
    s.set_mesh(cube)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    s.set_mesh(strip)
    torch.cuda.synchronize()
    assert torch.cuda.mem_get_info()[0] >= before
    for _ in range(2):
        s.upload_state(S)
        s.step(1e-6, 2)
        out.append(s.download_state())
        s.close()
        s = Solver(**args)
        s.set_mesh(strip)
    s.close()
    assert np.isfinite(out[0]).all()
    np.testing.assert_array_equal(out[0], out[1])
