"""Ghost-fluid fixes of many cells in one pass: a mixture whose solid fraction is within rounding
of AVF_LIM almost everywhere, so that a stage crosses it in hundreds of cells (ranked in shared
memory) or in thousands (collected from the flags).  The fixes run in leaf order and read earlier
neighbours' new states: the FP64 form against the CPU restatement of the reference, whose own
count of fixes must show that the case does what it is for.

The bar is the other parity tests' 1e-12 for all that the fixes write.  The volume fractions and
internal energies pass through the relaxation after them, whose iteration stops at |F| <= 1e-12: two
evaluations whose powers differ in the last bit may stop one iterate apart, a fraction then differs
by up to 1e-12, and the energy of the smallest fraction here, 0.1, by 1e-11 of itself."""
import numpy as np
import pytest

from forestfv_public_gb300 import Mesh, Solver, uniform_leaves
from forestfv_public_gb300 import workloads as W
from oracle import pyoracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("level,at_least", [(3, 100), (5, 10000)])
def test_many_crossings_match_oracle(level, at_least, built_lib, oracle_lib):
    mesh = Mesh((2, 2, 2), uniform_leaves((2, 2, 2), level))
    m = W.WALL
    rng = np.random.default_rng(11)
    n = mesh.n
    x = mesh.centroids()
    a0 = 0.5 + 1e-4 * np.sin(9.0 * x[:, 0]) * np.cos(7.0 * x[:, 1] + 3.0 * x[:, 2])
    a2 = np.full(n, 0.1)
    alpha = np.stack([a0, 1.0 - a0 - a2, a2])
    S = np.zeros((21, n))
    p = 5e6
    for k in range(3):
        S[k] = alpha[k] * m["rho"][k]
        S[9 + k] = alpha[k] * (p + m["gamma"][k] * m["pinf"][k]) / (m["gamma"][k] - 1.0)
    rho = S[:3].sum(0)
    S[3:6] = rho * 50.0 * np.stack([np.sin(11.0 * x[:, i] + i) for i in range(3)])
    S[6] = S[9:12].sum(0) + 0.5 * (S[3:6] ** 2).sum(0) / rho
    S[7], S[8] = alpha[0], alpha[1]
    for q in (0, 4, 8):
        S[12 + q] = 1.0
    S[0] *= 1.0 + 1e-3 * rng.uniform(-1, 1, n)
    dt = 0.02 * 0.5 / (1 << (level - 1)) / np.sqrt(3.5 * (5e6 + 3.2e10) / 2700.0)
    s = Solver(model=5, gamma=m["gamma"], pinf=m["pinf"], mu=m["mu"], amin=m["amin"], avf_lim=0.5,
               prelax=3, flux_form=1)
    s.set_mesh(mesh)
    s.upload_state(S)
    s.step(dt, 1)
    out = s.download_state()
    s.close()
    before = pyoracle.m5_gfm_calls()
    m5 = dict(avf_lim=0.5, prelax=3, amin=m["amin"], pinf=list(m["pinf"]), gamma=list(m["gamma"]),
              mu=list(m["mu"]), flux_form=1)
    ref = pyoracle.m5_advance(pyoracle.OracleMesh(mesh.export()), S.T.copy(), dt, 1, m5).T
    calls = np.subtract(pyoracle.m5_gfm_calls(), before)
    assert calls.max() >= at_least, calls
    scale = np.abs(ref).max(axis=1)
    err = np.abs(out - ref).max(axis=1) / np.maximum(scale, 1e-300)
    bar = np.full(21, 1e-12)
    bar[7:12] += 1e-12 / 0.1
    assert np.isfinite(out).all() and (err <= bar).all(), (err.max(), int(err.argmax()), calls)
