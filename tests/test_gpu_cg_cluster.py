"""The CG iteration in one cluster launch: one, two and four atoms a thread and
the first size beyond, the queued-ahead form, and the iteration limit.

A step of size eps in the Jacobi map leaves eps / (1 - spectral radius) of the
fixed point, at most ten times eps here: targets of 1e-10 e nm against dipoles of
1e-2 give 1e-7 relative RMS."""
import numpy as np
import pytest

from tholedipoleplugin_b200 import systems as S
from tholedipoleplugin_b200.kernel import CudaCalcTholeDipoleForceKernel

pytestmark = pytest.mark.gpu


def rel_rms(a, b):
    return float(np.sqrt(np.mean((a - b) ** 2) / np.mean(b ** 2)))


@pytest.mark.parametrize("n_side", [3, 7, 11, 12, 14, 17, 18])   # 4,096, 8,192 and 16,384 atoms lie in between
def test_agrees_with_jacobi(n_side):
    s = S.water_box(n_side, 0.3107 * n_side, seed=n_side, cutoff=0.4, target_eps=1e-10, max_iter=200)
    s = s.copy(polarizabilities=0.4 * s.polarizabilities)   # the Jacobi sweep contracts
    out = []
    for solver in ("cg", "jacobi"):
        with CudaCalcTholeDipoleForceKernel(s, precision="double", solver=solver) as k:
            out.append(k.getInducedDipoles(s.positions))
            assert k.solverStats()["converged"] == 1
    assert rel_rms(*out) < 1e-7


@pytest.mark.parametrize("n_side", [6, 11, 18])
@pytest.mark.parametrize("precision", ["mixed", "double"])
def test_iteration_limit(n_side, precision):
    s = S.water_box(n_side, 0.3107 * n_side, seed=1, cutoff=0.8, target_eps=1e-12)
    full = []
    for limit in (1, 2, 3):
        with CudaCalcTholeDipoleForceKernel(s.copy(max_iter=limit), precision=precision) as k:
            k.getInducedDipoles(s.positions)
            st = k.solverStats()
            assert st["iterations"] == limit and st["converged"] == 0
            full.append(st["epsilon"])
    assert full[0] > full[1] > full[2] > 0.0
