"""Model 0's face-once stage at the sizes and forests where it can go wrong: one cell, fewer
cells than a block, one more than a block, a cell edge that is no power of two (the limiter's
quotients instead of its bit form), hanging faces on every side of a cell, every boundary code,
both orders.  Bit-identical to the CPU restatement of the reference."""
import numpy as np
import pytest

from forestfv_public_gb300 import Mesh, Solver, uniform_leaves
from forestfv_public_gb300 import workloads as W
from oracle import pyoracle

pytestmark = pytest.mark.gpu


def shell(lmin, lmax, r):
    """A forest refined around a sphere, so that cells have coarser and finer neighbours on
    several sides."""
    def target(cen, h):
        d = np.abs(np.linalg.norm(cen - 0.5, axis=1) - r) - 0.87 * h
        return np.where(d < 0.02, lmax, lmin)
    return W.refine_to_target((2, 2, 2), lmin, lmax, target)


CASES = {
    "one_cell": ((1, 1, 1), 1, 1.0),
    "row_of_five": ((5, 1, 1), 1, 0.25),
    "block_and_one": ((43, 3, 1), 1, 0.5),   # 129 cells
    "edge_not_a_power_of_two": ((3, 2, 1), 3, 0.75),
    "hanging": None,
}


@pytest.mark.parametrize("order,rk,bc", [(2, 2, 2), (1, 3, 4), (2, 4, 5), (2, 1, 1)])
@pytest.mark.parametrize("case", sorted(CASES))
def test_stage_matches_oracle(case, order, rk, bc, built_lib, oracle_lib):
    if CASES[case] is None:
        mesh = Mesh((2, 2, 2), shell(3, 4, 0.3), bc=(bc,) * 6)
    else:
        trees, level, edge = CASES[case]
        mesh = Mesh(trees, uniform_leaves(trees, level), bc=(bc,) * 6, tree_edge=edge)
    rng = np.random.default_rng(7)
    S = np.empty((5, mesh.n))
    S[0] = rng.uniform(0.5, 2.0, mesh.n)
    S[1:4] = S[0] * rng.uniform(-0.5, 0.5, (3, mesh.n))
    S[4] = rng.uniform(1.0, 3.0, mesh.n) / 0.4 + 0.5 * (S[1:4] ** 2).sum(0) / S[0]
    S[:, ::3] = S[:, :1]  # equal neighbours here and there: no slope
    dt = 0.05 * float(mesh.tree_edge / (1 << (int(mesh.level.max()) - 1)))
    s = Solver(model=0, order=order, rk_steps=rk)
    s.set_mesh(mesh)
    s.upload_state(S)
    s.step(dt, 3)
    out = s.download_state()
    s.close()
    ref = pyoracle.m0_advance(pyoracle.OracleMesh(mesh.export()), S.T.copy(), dt, 3, order=order,
                              rk_steps=rk).T
    assert np.array_equal(out, ref), np.abs(out - ref).max()
