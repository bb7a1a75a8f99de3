"""Model 5's FP64 stage on forests where its bit-level forms give way to the plain ones: a cell
edge that is no power of two, one cell, a row of cells, boundary cells on every side, hanging
faces; both flux forms and orders, against the CPU restatement of the reference to 1e-12 of each
variable's largest value (the reference form's arithmetic is the restatement's but for the last
bit of pow; the bar is the one of the other parity tests)."""
import numpy as np
import pytest

from forestfv_public_gb300 import Mesh, Solver, uniform_leaves
from forestfv_public_gb300 import workloads as W
from oracle import pyoracle

pytestmark = pytest.mark.gpu

CASES = {"one_cell": ((1, 1, 1), 1, 1.0), "row": ((7, 1, 1), 1, 0.125), "three_quarters": ((3, 2, 2), 2, 0.75),
         "long_row": ((3000, 1, 1), 1, 0.125),  # more boundary faces than cells
         "hanging": None}


def shell():
    def target(cen, h):
        d = np.abs(np.linalg.norm(cen - 0.5, axis=1) - 0.3) - 0.87 * h
        return np.where(d < 0.02, 4, 3)
    return W.refine_to_target((2, 2, 2), 3, 4, target)


@pytest.mark.parametrize("flux_form", [0, 1])
@pytest.mark.parametrize("order,rk,bc", [(2, 2, 2), (2, 3, 4), (1, 2, 5), (2, 2, 1)])
@pytest.mark.parametrize("case", sorted(CASES))
def test_fp64_stage_matches_oracle(case, order, rk, bc, flux_form, built_lib, oracle_lib):
    if CASES[case] is None:
        mesh = Mesh((2, 2, 2), shell(), bc=(bc,) * 6)
    else:
        trees, level, edge = CASES[case]
        mesh = Mesh(trees, uniform_leaves(trees, level), bc=(bc,) * 6, tree_edge=edge)
    m = W.WALL
    x = mesh.centroids()
    x = x / x.max()
    S = W.wall_state(m, x[:, 2] < 0.25, 0.5 - 0.4 * np.cos(5.0 * x[:, 0]))
    h = mesh.tree_edge / (1 << (int(mesh.level.max()) - 1))
    dt = 0.01 * h / np.sqrt(3.5 * (5e6 + 3.2e10) / 2700.0)
    s = Solver(model=5, order=order, rk_steps=rk, gamma=m["gamma"], pinf=m["pinf"], mu=m["mu"],
               amin=m["amin"], avf_lim=m["avf_lim"], prelax=3, flux_form=flux_form)
    s.set_mesh(mesh)
    s.upload_state(S)
    s.step(dt, 2)
    out = s.download_state()
    s.close()
    m5 = dict(avf_lim=m["avf_lim"], prelax=3, amin=m["amin"], pinf=list(m["pinf"]),
              gamma=list(m["gamma"]), mu=list(m["mu"]), flux_form=flux_form)
    ref = pyoracle.m5_advance(pyoracle.OracleMesh(mesh.export()), S.T.copy(), dt, 2, m5, order=order,
                              rk_steps=rk).T
    scale = np.maximum(np.abs(ref).max(axis=1), 1e-300)
    # a momentum that only rounding moves is measured against what the pressures could give it
    scale[3:6] = np.maximum(scale[3:6], 5e6 * dt / h)
    err = np.abs(out - ref).max(axis=1) / scale
    assert np.isfinite(out).all() and (err <= 1e-12).all(), (err.max(), int(err.argmax()))
