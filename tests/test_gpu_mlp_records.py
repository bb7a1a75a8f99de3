"""The indicator's feature rows on a mesh against rows put together on the host from the same fields:
each value normalised in FP32 and rounded to BF16 (ties to even), the 27 stencil cells in order.  Both
do the same two FP32 operations and one rounding, so the rows are equal bit by bit.  Blocks end in the
middle of the mesh (1576, 5 and 240 cells); boundaries and hanging faces are among the stencils."""
import numpy as np
import pytest
import torch

from forestfv_public_gb300 import Mesh, Solver, uniform_leaves
from forestfv_public_gb300 import workloads as W
from forestfv_public_gb300.indicator import Indicator
from oracle import mlp
from test_gpu_m5_forests import shell

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["hanging", "row", "box"])
def test_rows_equal_host_rows(name, built_lib):
    mesh = {"hanging": lambda: Mesh((2, 2, 2), shell(), bc=(2,) * 6),
            "row": lambda: Mesh((5, 1, 1), uniform_leaves((5, 1, 1), 1), bc=(2,) * 6),
            "box": lambda: Mesh((5, 3, 2), uniform_leaves((5, 3, 2), 2), bc=(2,) * 6)}[name]()
    m = W.WALL
    x = mesh.centroids()
    S = W.wall_state(m, x[:, 2] < 0.3 * x.max(), 0.5 - 0.4 * np.cos(5.0 * x[:, 0]))
    s = Solver(model=5, order=2, rk_steps=2, gamma=m["gamma"], pinf=m["pinf"], mu=m["mu"], amin=m["amin"],
               avf_lim=m["avf_lim"], prelax=3)
    s.set_mesh(mesh)
    s.upload_state(S)
    ind = Indicator(seed=3)
    F = ind.fields(s).cpu().numpy()
    mean, std = F.mean(axis=1), F.std(axis=1) + np.float32(1e-3)
    ind.set_norm(mean, std)
    X = ind.features(s).float().cpu().numpy()[:, :mlp.NIN]
    V = (F - mean[:, None]) * (np.float32(1.0) / std)[:, None]
    assert V.dtype == np.float32
    V = torch.from_numpy(V).to(torch.bfloat16).double().numpy()
    ref = mlp.stencil_features(mesh.export(), V, np.zeros(5), np.ones(5))
    np.testing.assert_array_equal(X, ref)
    assert np.array_equal(ind.predict(s), ind.forward(ind.features(s)).cpu().numpy())
    ind.close()
    s.close()
