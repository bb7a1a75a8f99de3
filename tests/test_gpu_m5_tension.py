"""Pressure relaxation of the FP32-flux form where the mean pressure lies below the gas's bound (a
liquid under tension beside a little gas), which starts its Newton iteration from a bound of the
root, against the FP64 form.  The equilibrium pressure is found to 1e-7 of itself or to F's rounding,
6e-8 of a unit sum over the sum's slope; the fractions of the two forms then agree to 2e-6 of the
smaller one, the internal energies to 2e-6 of their sum."""
import numpy as np
import pytest

from forestfv_public_gb300 import Mesh, Solver, uniform_leaves
from forestfv_public_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("liquid", [-1e3, -4.4e5, -5.3e6, -4e7])
@pytest.mark.parametrize("gas", [1e5, 7.1e6])
def test_relaxation_under_tension(liquid, gas, built_lib):
    mesh = Mesh((1, 1, 1), uniform_leaves((1, 1, 1), 3), bc=(2,) * 6)
    m = W.WALL
    frac = np.geomspace(2e-5, 0.6, mesh.n)
    a = np.stack([np.full(mesh.n, 1e-6), 1.0 - 1e-6 - frac, frac])
    p = np.stack([np.full(mesh.n, 5e6), np.full(mesh.n, liquid), np.full(mesh.n, gas)])
    g, pi, rho = (np.array(m[q])[:, None] for q in ("gamma", "pinf", "rho"))
    S = np.zeros((21, mesh.n))
    S[:3] = a * rho
    S[7:9] = a[:2]
    S[9:12] = a * (p + g * pi) / (g - 1.0)
    S[6] = S[9:12].sum(axis=0)
    out = []
    for precision in (0, 1):
        s = Solver(model=5, order=1, rk_steps=2, gamma=m["gamma"], pinf=m["pinf"], mu=m["mu"], amin=m["amin"],
                   avf_lim=m["avf_lim"], prelax=3, flux_form=1, precision=precision)
        s.set_mesh(mesh)
        s.upload_state(S)
        s.step(1e-16, 1)
        out.append(s.download_state())
        s.close()
    ref, got = out
    assert np.isfinite(got).all() and np.abs(ref[8] - S[8]).max() > 1e-6  # it did relax
    rest = np.minimum(ref[8], 1.0 - ref[7] - ref[8])
    assert (np.abs(got[8] - ref[8]) <= 2e-6 * rest).all(), (np.abs(got[8] - ref[8]) / rest).max()
    assert (np.abs(got[9:12] - ref[9:12]) <= 2e-6 * ref[6]).all()
