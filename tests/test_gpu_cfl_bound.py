"""The CFL step where cells are passed over (meshes of more cells than the kernel has threads): a cell
may be left out only if it is certainly slower than one already seen and certainly has a speed.

A gas beside a trace of a stiff last material: c^2 is what remains of that material's energy and
p_inf, so the fraction's rounding counts.  The fastest cells come second in every thread, their
fractions chosen so that 1 - alpha in FP32 makes them look slower than the first; the result against
the plain formula in numpy, to 1e-14 as in test_gpu_tags_edges (the sum cancels by ~4 here too).
And cells without a speed beside faster ones: a momentum or a solid's deformation that is not a
number, and a c^2 that the elastic energy alone makes negative."""
import numpy as np
import pytest

from forestfv_public_gb300 import Mesh, Solver, uniform_leaves
from forestfv_public_gb300 import workloads as W
from forestfv_public_gb300._lib import FFVError

pytestmark = pytest.mark.gpu
FIRST = 152 * 4 * 128  # threads: cell c and c + FIRST are seen by one
FFV_ERR_NAN = 5


@pytest.fixture(scope="module")
def mesh():
    return Mesh((2, 2, 2), uniform_leaves((2, 2, 2), 6))


@pytest.mark.parametrize("gamma,pinf,p", [([1.4, 3.5], [0.0, 3.2e10], 1e5), ([1.4, 4.4], [0.0, 6e8], 1e4),
                                          ([1.4, 1.4, 3.5], [0.0, 0.0, 7e10], 1e5)])
@pytest.mark.parametrize("seed", [1, 2])
def test_stiff_trace_beside_gas(gamma, pinf, p, seed, mesh, built_lib):
    rng = np.random.default_rng(seed)
    n, N = mesh.n, len(gamma)
    assert n > 2 * FIRST
    seen_first = np.arange(n) < FIRST
    # FP32 values of the gas's fraction(s), but for the later cells almost half an ulp above one:
    # rounded down again, which makes the last fraction look 2.7e-8 larger
    share = np.ones(n) if N == 2 else rng.uniform(0.9, 0.99, n)
    alpha = [((1.0 - 1e-6) * share).astype(np.float32) + np.where(seen_first, 0.0, 0.45 * 2.0 ** -24)]
    if N == 3:
        alpha.append((1.0 - 1e-6 - alpha[0]).astype(np.float32).astype(np.float64))
    alpha.append(1.0 - alpha[0] if N == 2 else 1.0 - (alpha[0] + alpha[1]))
    assert (alpha[-1] > 5e-7).all()
    energy = [alpha[k] * (p + gamma[k] * pinf[k]) / (gamma[k] - 1.0) for k in range(N)]
    rho_c2 = sum(gamma[k] * (gamma[k] - 1.0) * (energy[k] - alpha[k] * pinf[k]) for k in range(N))
    # sound speeds: the cells each thread sees first a little slower than the others
    rho = rho_c2 / (400.0 * np.where(seen_first, 1.0, 1.004 + 1e-4 * rng.random(n))) ** 2
    S = np.zeros((3 * N + 12, n))
    for k in range(N):
        S[k] = alpha[k] * rho
        S[2 * N + 3 + k] = energy[k]
    for k in range(N - 1):
        S[N + 4 + k] = alpha[k]
    S[N:N + 3] = rho * rng.uniform(-0.1, 0.1, (3, n))
    S[N + 3] = sum(energy)
    r = sum(S[:N])
    want = 0.3 * (0.5 / 2.0 ** 5) / (np.abs(S[N:N + 3] / r).max(0) + np.sqrt(rho_c2 / r)).max()
    s = Solver(model=5, gamma=gamma, pinf=pinf, mu=[0.0] * N, amin=1e-6, avf_lim=0.5, prelax=3, flux_form=1)
    s.set_mesh(mesh)
    s.upload_state(S)
    got = s.cfl_dt(0.3)
    s.close()
    assert abs(got - want) <= 1e-14 * want, got / want - 1.0


@pytest.mark.parametrize("what", ["momentum", "deformation", "elastic energy", "elastic energy of a small strain",
                                  "nothing"])
def test_cells_without_a_speed(what, mesh, built_lib):
    m, n = W.WALL, mesh.n
    S = W.wall_state(m, np.arange(n) < FIRST + 100, np.zeros(n))  # solid first, liquid after
    c = n - 77
    if what == "momentum":
        S[4, c] = np.nan
    elif what == "deformation":
        S[12:, c] = np.array([1, 0, 0, 0, 1, 0, 0, 0, 1.0])
        S[14, c] = np.nan
    elif what == "elastic energy":
        S[12:, c] = np.array([2, 0, 0, 0, 1, 0, 0, 0, 1.0])
    elif what == "elastic energy of a small strain":
        # eps = 0.02: e_el is several MPa, which the energies just miss
        S[12:, c] = np.array([1.01, 0, 0, 0, 1, 0, 0, 0, 1.0])
        g, p = m["gamma"], m["pinf"]
        al = [S[7, c], S[8, c], 1.0 - S[7, c] - S[8, c]]
        for k in range(3):
            S[9 + k, c] = al[k] * p[k] + 1e4
    s = Solver(model=5, gamma=m["gamma"], pinf=m["pinf"], mu=m["mu"], amin=m["amin"], avf_lim=0.5, prelax=3,
               flux_form=1)
    s.set_mesh(mesh)
    s.upload_state(S)
    if what == "nothing":
        assert s.cfl_dt(0.3) > 0.0
    else:
        with pytest.raises(FFVError) as e:
            s.cfl_dt(0.3)
        assert e.value.code == FFV_ERR_NAN
    s.close()
