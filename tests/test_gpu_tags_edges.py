"""The criterion's screens and lists at their edges, against the oracle's restatement of the
reference's tags: density and pressure jumps within 1e-7 of the threshold and exactly on it, zero
and negative thresholds, many interface layers on a mesh with hanging faces (both volume
fractions), solid fractions exactly at AVF_LIM, and a part of a forest, whose neighbour relation is
not symmetric.  Identical tags.  And the CFL step at cells that its screen passes over, against the
plain formula in numpy."""
import numpy as np
import pytest

from forestfv_public_gb300 import Mesh, Solver
from forestfv_public_gb300 import workloads as W
from forestfv_public_gb300.mesh import Leaves
from oracle import tags as T

pytestmark = pytest.mark.gpu
M = dict(W.WALL)
M5 = dict(avf_lim=0.5, amin=M["amin"], gamma=list(M["gamma"]), pinf=list(M["pinf"]), mu=list(M["mu"]), prelax=3)


def leaves():
    def target(cen, h):
        d = np.abs(np.linalg.norm(cen - 0.5, axis=1) - 0.25) - 0.87 * h
        return np.where(d < 0.03, 5, np.where(d < 0.2, 4, 3))
    return W.refine_to_target((2, 2, 2), 3, 5, target)


def state(mesh, seed):
    rng = np.random.default_rng(seed)
    x = mesh.centroids()
    r = np.linalg.norm(x - 0.5, axis=1)
    S = W.wall_state(M, x[:, 2] < 0.3, 0.5 - 0.5 * np.tanh((r - 0.25) / 0.02))
    S[7] = np.where(rng.random(mesh.n) < 0.02, 0.5, S[7])  # exactly AVF_LIM here and there
    # densities on a few values whose relative jumps lie on and beside 0.1
    top = np.array([1.0, 1.0 / 0.9, 1.0 / (0.9 * (1 + 3e-8)), 1.0 / (0.9 * (1 - 3e-8)), 1.0 / (0.9 + 1e-16), 1.3])
    S[:3] *= (1000.0 * top[rng.integers(0, 6, mesh.n)] / S[:3].sum(0))
    return S


def solver(mesh, S):
    s = Solver(model=5, gamma=M["gamma"], pinf=M["pinf"], mu=M["mu"], amin=M["amin"], avf_lim=0.5, prelax=3,
               flux_form=1)
    s.set_mesh(mesh)
    s.upload_state(S)
    return s


PARAMS = [(1, 3, 1, 5, 0.1, 1, 5, 0.1, 0, 0, 0.0, 1, 5, 9, 0, 0, 0),
          (1, 3, 0, 0, 0.0, 1, 4, 0.1, 1, 5, 0.3, 1, 4, 3, 1, 5, 12),
          (1, 3, 1, 4, 0.0, 1, 5, -1.0, 0, 0, 0.0, 1, 5, 2, 0, 0, 0),
          (0, 3, 0, 0, 0.0, 1, 5, 0.10000003, 0, 0, 0.0, 0, 0, 0, 0, 0, 0)]


@pytest.mark.parametrize("part", [False, True])
@pytest.mark.parametrize("seed", [1, 2])
def test_tags_match_oracle(seed, part, built_lib):
    lv = leaves()
    if part:  # drop an eighth of the fine leaves: some coarse cells lose a finer neighbour
        keep = ~((lv.level == 5) & (lv.cell_ijk.sum(1) % 8 == 3))
        lv = Leaves(lv.tree_ijk[keep], lv.level[keep], lv.cell_ijk[keep])
    mesh = Mesh((2, 2, 2), lv, part=part)
    S = state(mesh, seed)
    s = solver(mesh, S)
    ex = mesh.export()
    for p in PARAMS:
        split, raw, si = s.tags(p, with_raw=True)
        SI = T.interface_layers(S, ex, M5, T.si_max(p)) if p[11] else np.zeros((2, mesh.n), np.int32)
        assert np.array_equal(si, SI), p
        assert np.array_equal(raw, T.raw_levels(S, ex, M5, p, SI)), p
        assert s.tags_missed(p) == int((raw > mesh.level).sum()), p
    s.close()


def test_cfl_step(built_lib):
    mesh = Mesh((2, 2, 2), leaves())
    S = state(mesh, 3)
    x = mesh.centroids()
    a = S[7:9].copy()
    al = np.stack([a[0], a[1], 1.0 - a[0] - a[1]]).clip(M["amin"] / 100.0, 1.0)
    rho = S[:3].sum(0)
    S[3:6] = rho * 100.0 * np.sin(7.0 * x.T)
    c2 = sum(al[k] / rho * M["gamma"][k] * ((M["gamma"][k] - 1.0) * S[9 + k] / al[k] - M["gamma"][k] * M["pinf"][k]
                                           + M["pinf"][k]) for k in range(3))
    ok = c2 > 0  # a fraction set to AVF_LIM beside energies of a fluid may have none
    S[7:9] = np.where(ok, S[7:9], W.wall_state(M, np.ones(mesh.n, bool), np.zeros(mesh.n))[7:9])
    S[9:12] = np.where(ok, S[9:12], W.wall_state(M, np.ones(mesh.n, bool), np.zeros(mesh.n))[9:12])
    S[12:] = 0.0
    al = np.stack([S[7], S[8], 1.0 - S[7] - S[8]]).clip(M["amin"] / 100.0, 1.0)
    c2 = sum(al[k] / rho * M["gamma"][k] * ((M["gamma"][k] - 1.0) * S[9 + k] / al[k] - M["gamma"][k] * M["pinf"][k]
                                           + M["pinf"][k]) for k in range(3))
    h = 0.5 / 2.0 ** (mesh.level - 1)
    want = 0.3 * (h / (np.abs(S[3:6] / rho).max(0) + np.sqrt(c2))).min()
    s = solver(mesh, S)
    got = s.cfl_dt(0.3)
    s.close()
    # the sum cancels by at most ~4: a few units in the last place of c^2, half of that in c
    assert abs(got - want) <= 1e-14 * want
