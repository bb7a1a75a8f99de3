"""The FP32-flux form's marks of cells without deformation (fluid, A = 0): a marked state is carried
without its deformation, an unmarked one in full.  The same fluid with A = 1e-300 (not marked; its
FP32 deviation from the identity is the same -1) takes the full path, and one step of both has to
agree: every value within 2e-6 of its variable's largest (the paths differ by the FP32 rounding of
the star deformation, 6e-8 of 1 times a Courant number of 0.1, and by how products contract: a few
6e-8 of each flux).  Fluid out of the solid's reach stays at A = 0 to the bit, and a step by stages,
whose marks come from the state, equals the captured step, whose later stages keep them."""
import numpy as np
import pytest

from forestfv_public_gb300 import Mesh, Solver, uniform_leaves
from forestfv_public_gb300 import workloads as W
from test_gpu_m5_forests import shell

pytestmark = pytest.mark.gpu


def case(name, bc, mesh=None):
    if mesh is not None:
        pass
    elif name == "hanging":
        mesh = Mesh((2, 2, 2), shell(), bc=(bc,) * 6)
    else:
        mesh = Mesh((2, 2, 12), uniform_leaves((2, 2, 12), 2), bc=(bc,) * 6)
    m = W.WALL
    x = mesh.centroids()
    x = x / x.max()
    S = W.wall_state(m, x[:, 2] < 0.3, 0.5 - 0.4 * np.cos(5.0 * x[:, 0]))
    vel = np.stack([30.0 * np.sin(3.0 * x[:, 1]), 20.0 * np.cos(2.0 * x[:, 0]), 40.0 * np.cos(7.0 * x[:, 0])])
    rho = S[:3].sum(axis=0)
    S[3:6] = rho * vel
    S[6] += 0.5 * rho * (vel ** 2).sum(axis=0)
    h = mesh.tree_edge / (1 << int(mesh.level.max()))
    return mesh, m, S, 0.1 * h / np.sqrt(3.5 * (5e6 + 3.2e10) / 2700.0)


def solver(mesh, m, S, order, rk, **kw):
    s = Solver(model=5, order=order, rk_steps=rk, gamma=m["gamma"], pinf=m["pinf"], mu=m["mu"],
               amin=m["amin"], avf_lim=m["avf_lim"], prelax=3, flux_form=1, precision=1, **kw)
    s.set_mesh(mesh)
    s.upload_state(S)
    return s


@pytest.mark.parametrize("name,bc,order,rk", [("hanging", 2, 2, 2), ("hanging", 1, 2, 3), ("uniform", 4, 2, 2),
                                              ("uniform", 5, 2, 2), ("hanging", 2, 1, 2)])
def test_marked_fluid_against_full_path(name, bc, order, rk, built_lib):
    mesh, m, S, dt = case(name, bc)
    fluid = (S[-9:] == 0.0).all(axis=0)
    assert fluid.any() and not fluid.all()
    T = S.copy()
    T[-9:, fluid] = 1e-300
    out = []
    for U in (S, T):
        s = solver(mesh, m, U, order, rk)
        s.step(dt, 1)
        out.append(s.download_state())
        s.close()
    assert np.isfinite(out[0]).all()
    scale = np.abs(out[1]).max(axis=1, keepdims=True)
    scale[3:6] = np.maximum(scale[3:6], 1.0)
    scale[-9:] = 1.0
    err = (np.abs(out[0] - out[1]) / scale).max(axis=1)
    assert (err <= 2e-6).all(), err


@pytest.mark.parametrize("name,order,rk", [("hanging", 2, 2), ("uniform", 2, 3), ("uniform", 1, 2)])
def test_fluid_out_of_reach_and_stages(name, order, rk, built_lib):
    mesh, m, S, dt = case(name, 2)
    S[-9:, :1] = -0.0  # a zero of either sign is none
    s = solver(mesh, m, S, order, rk)
    s.step(dt, 2)
    out = s.download_state()
    s.close()
    cen = mesh.centroids()
    solid = cen[(S[-9:] != 0.0).any(axis=0)]
    h = mesh.tree_edge / (1 << (int(mesh.level.min()) - 1))
    far = cen[:, 2] > solid[:, 2].max() + (2 * rk + 0.5) * h
    assert (far.any() or name == "hanging") and not out[-9:, far].any()
    s = solver(mesh, m, S, order, rk)
    for _ in range(2):
        for irk in range(1, rk + 1):
            s.rk(irk, dt)
    s.sync()
    again = s.download_state()
    s.close()
    np.testing.assert_array_equal(again, out)


def large(name):
    """meshes of more than the 456 blocks from which warps of unmarked surroundings go their own way"""
    if name == "hanging":  # a shell two levels deep that crosses the solid's surface
        def target(cen, h):
            return np.where(np.abs(np.linalg.norm(cen - 0.5, axis=1) - 0.3) < 0.06, 6, 5)
        return Mesh((2, 2, 2), W.refine_to_target((2, 2, 2), 5, 6, target), bc=(2,) * 6)
    return Mesh((3, 3, 13), uniform_leaves((3, 3, 13), 4), bc=(2,) * 6)  # 59,904 cells: 468 blocks


@pytest.mark.parametrize("name,rk", [("hanging", 2), ("hanging", 3), ("uniform", 2)])
def test_calm_warps_against_full_path(name, rk, built_lib):
    mesh = large(name)
    assert mesh.n > 456 * 128
    m, S, dt = case("uniform", 2, mesh)[1:]
    T = S.copy()
    T[-9:, (S[-9:] == 0.0).all(axis=0)] = 1e-300
    out = []
    for U in (S, T):
        s = solver(mesh, m, U, 2, rk)
        s.step(dt, 1)
        out.append(s.download_state())
        s.close()
    scale = np.abs(out[1]).max(axis=1, keepdims=True)
    scale[3:6] = np.maximum(scale[3:6], 1.0)
    scale[-9:] = 1.0
    err = (np.abs(out[0] - out[1]) / scale).max(axis=1)
    assert np.isfinite(out[0]).all() and (err <= 2e-6).all(), err
