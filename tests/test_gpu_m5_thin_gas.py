"""The consistent form's FP64 relaxation where a material has almost no mass left.  A gas of 2^-110 kg/m^3
beside a liquid is too thin to show in any sum of densities, and its slopes are below the limiter's
threshold: thinning it by another power of two scales its partial density, divides every quotient of
two such densities out, and changes no other bit.  Down to 2^-910, far below what an FP32 reciprocal
resolves.  Two steps: identical bits, the gas's own partial density scaled."""
import numpy as np
import pytest

from forestfv_public_gb300 import Mesh, Solver, uniform_leaves
from forestfv_public_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def advance(thin):
    mesh = Mesh((2, 2, 2), uniform_leaves((2, 2, 2), 3))
    m = W.BUBBLE
    x = mesh.centroids() / mesh.centroids().max()
    gas = np.clip(0.5 - 0.6 * np.cos(4.0 * x[:, 0] + x[:, 1]), 1e-6, 1.0 - 1e-6)
    alpha = np.stack([1.0 - gas, gas])
    p = 1e5 * (1.0 + 0.1 * np.sin(7.0 * x[:, 1]))
    S = np.zeros((18, mesh.n))
    for k, rho in enumerate((1000.0, thin)):
        S[k] = alpha[k] * rho
        S[7 + k] = alpha[k] * (p + m["gamma"][k] * m["pinf"][k]) / (m["gamma"][k] - 1.0)
    r = S[0] + S[1]
    S[2:5] = r * 5.0 * np.stack([np.sin(11.0 * x[:, i] + i) for i in range(3)])
    S[5] = S[7] + S[8] + 0.5 * (S[2:5] ** 2).sum(0) / r
    S[6] = alpha[0]
    s = Solver(model=5, gamma=m["gamma"], pinf=m["pinf"], mu=m["mu"], amin=m["amin"], prelax=3, flux_form=1)
    s.set_mesh(mesh)
    s.upload_state(S)
    s.step(1e-4 * mesh.tree_edge / 4.0 / 1630.0, 2)
    out = s.download_state()
    s.close()
    return out


@pytest.mark.parametrize("power", [15, 20, 60, 400, 800])
def test_thinner_gas(power, built_lib):
    want, got = advance(2.0 ** -110), advance(2.0 ** -(110 + power))
    assert np.isfinite(want).all() and (want[1] > 0.0).all()
    want[1] *= 2.0 ** -power
    np.testing.assert_array_equal(got, want)
