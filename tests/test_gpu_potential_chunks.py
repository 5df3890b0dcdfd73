"""The potential query's split of points into blocks and atoms into chunks, at
the edges of both (one point, a block of 128 and its neighbours, systems below
and just above one staged step of 128 atoms), against the FP64 oracle.

Direct polarization keeps the solver out of it, so only the order of at most
n FP64 additions differs from the oracle: 1e-12 of the largest potential is
n eps with a factor of ten to spare at n = 1029."""
import numpy as np
import pytest

from oracle import oracle as O
from tholedipoleplugin_b200 import systems as S
from tholedipoleplugin_b200.kernel import CudaCalcTholeDipoleForceKernel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_side,method", [(3, S.NO_CUTOFF), (6, S.PME), (7, S.PME)])
@pytest.mark.parametrize("points", [1, 127, 128, 129, 1000])
def test_potential_blocks_and_chunks(n_side, method, points):
    s = S.water_box(n_side, 0.3107 * n_side, seed=n_side, cutoff=0.8, polarization=S.DIRECT, method=method)
    rng = np.random.default_rng(points)
    edge = 0.3107 * n_side
    grid = rng.uniform(-0.5 * edge, 1.5 * edge, size=(points, 3))
    # one point exactly half a box from an atom in x: the reference's floor(d/L + 0.5) decides the image
    grid[0] = s.positions[0] + np.array([0.5 * edge, 0.21, 0.0])
    ref = O.potential(s, grid, "port")
    with CudaCalcTholeDipoleForceKernel(s, precision="double") as k:
        got = k.getElectrostaticPotential(grid, s.positions)
    assert np.max(np.abs(got - ref)) <= 1e-12 * np.max(np.abs(ref))


@pytest.mark.parametrize("waters", [42, 43, 85, 86])   # 126, 129, 255, 258 atoms: one, two and three staged steps
@pytest.mark.parametrize("points", [1, 300])
def test_potential_about_one_staged_step(waters, points):
    s = S.water_cluster(waters, np.random.default_rng(waters), polarization=S.DIRECT)
    grid = np.random.default_rng(points).uniform(-0.5, 2.5, size=(points, 3))
    ref = O.potential(s, grid, "port")
    with CudaCalcTholeDipoleForceKernel(s, precision="double") as k:
        got = k.getElectrostaticPotential(grid, s.positions)
    assert np.max(np.abs(got - ref)) <= 1e-12 * np.max(np.abs(ref))
