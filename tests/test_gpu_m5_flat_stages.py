"""The FP32-flux form's marks on meshes beyond one wave, where warps of cells without deformation go
their own way: two captured steps (later stages keep the update's marks, whose cells' deformation
is stored nowhere but in the state) against the same steps by stages (marks from the state each time),
to the bit; and fluid out of the solid's reach stays at A = 0."""
import numpy as np
import pytest

from test_gpu_m5_flat import case, large, solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,rk", [("hanging", 2), ("hanging", 3), ("uniform", 2), ("uniform", 3)])
def test_captured_steps_equal_stages(name, rk, built_lib):
    mesh = large(name)
    assert mesh.n > 456 * 128
    m, S, dt = case("uniform", 2, mesh)[1:]
    s = solver(mesh, m, S, 2, rk)
    s.step(dt, 2)
    out = s.download_state()
    s.close()
    cen = mesh.centroids()
    solid = cen[(S[-9:] != 0.0).any(axis=0)]
    h = mesh.tree_edge / (1 << (int(mesh.level.min()) - 1))
    far = cen[:, 2] > solid[:, 2].max() + (2 * rk + 0.5) * h
    assert far.sum() > 1000 and not out[-9:, far].any()
    s = solver(mesh, m, S, 2, rk)
    for _ in range(2):
        for irk in range(1, rk + 1):
            s.rk(irk, dt)
    s.sync()
    again = s.download_state()
    s.close()
    assert np.isfinite(out).all()
    np.testing.assert_array_equal(again, out)
