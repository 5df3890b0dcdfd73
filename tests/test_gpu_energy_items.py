"""The mixed form's energy items: tile edges, partners with every scale, atoms
whose spatial order differs from their index order (either orientation of a
pair), pairs on and near the x axis, the 1/r^4 option.

Tolerances are the mixed form's: forces 2e-5 relative RMS, energy
1e-6 |E| + 3e-7 sqrt(sum (q_i q_j / r_ij)^2).  Near the axis the frame's X row
turns with the direction of (d_y, d_z), so coordinates rounded by 1e-7 nm give
1e-7 / 2e-3 of the closest pairs' forces: 1e-4 there."""
import numpy as np
import pytest

from oracle import oracle as O
from tholedipoleplugin_b200 import systems as S
from tholedipoleplugin_b200.kernel import CudaCalcTholeDipoleForceKernel

from . import fixtures as F

pytestmark = pytest.mark.gpu


def rel_rms(a, b):
    return float(np.sqrt(np.mean((a - b) ** 2) / np.mean(b ** 2)))


def energy_scale(s):
    d = s.positions[:, None] - s.positions[None]
    if s.method == S.PME:
        d -= s.box * np.floor(d / s.box + 0.5)
    r2 = (d ** 2).sum(-1)
    i, j = np.triu_indices(s.n, 1)
    return float(np.sqrt(((s.charges[i] * s.charges[j]) ** 2 / r2[i, j]).sum()))


def check(s, tol=2e-5, **kw):
    ref = O.compute(s.copy(target_eps=1e-12, max_iter=5000), "port") if not kw else None
    with CudaCalcTholeDipoleForceKernel(s, precision="mixed", **kw) as k:
        e, f = k.execute(s.positions)
    if ref is None:
        with CudaCalcTholeDipoleForceKernel(s, precision="double", **kw) as k:
            e0, f0 = k.execute(s.positions)
    else:
        e0, f0 = ref.energy, ref.forces
    assert rel_rms(f, f0) < tol
    assert abs(e - e0) < 1e-6 * abs(e0) + 3e-7 * energy_scale(s)


@pytest.mark.parametrize("n", [4, 31, 33, 64, 97])
@pytest.mark.parametrize("method", [S.NO_CUTOFF, S.PME])
@pytest.mark.parametrize("polarization", [S.DIRECT, S.MUTUAL, S.EXTRAPOLATED])
def test_tile_edges_scales_and_orientation(n, method, polarization):
    # random positions: the index order is as good as shuffled against the spatial one
    s = F.small_random_system(n, seed=100 + n, method=method, polarization=polarization, box=3.0)
    s = s.copy(polarizabilities=0.1 * s.polarizabilities, target_eps=1e-9, max_iter=2000)
    check(s)


@pytest.mark.parametrize("method", [S.NO_CUTOFF, S.PME])
def test_general_walk_matches_plain_form(method):
    s = F.small_random_system(97, seed=5, method=method, box=3.0)
    check(s.copy(polarizabilities=0.1 * s.polarizabilities, target_eps=1e-9, max_iter=2000), dd_force_r4=True)


@pytest.mark.parametrize("off,tol", [(0.0, 2e-5), (2e-3, 1e-4)])
@pytest.mark.parametrize("n", [70])
def test_pairs_on_and_near_the_x_axis(off, tol, n):
    rng = np.random.default_rng(n)
    pos = np.zeros((n, 3))
    pos[:, 0] = 0.31 * rng.permutation(n)
    pos[:, 1] = off * rng.choice([-1.0, 0.0, 1.0], n)
    pos[:, 2] = off * rng.choice([-1.0, 0.0, 1.0], n)
    axis = np.full((n, 4), -1, dtype=np.int32)
    axis[:, 0] = S.NOAXISTYPE
    s = S.TholeSystem(positions=pos, charges=rng.normal(scale=0.4, size=n), dipoles=rng.normal(scale=0.01, size=(n, 3)),
                      polarizabilities=rng.uniform(0.3e-3, 1.5e-3, n), tholes=rng.uniform(0.3, 0.45, n), axis=axis,
                      cov12=[[] for _ in range(n)], cov13=[[] for _ in range(n)], target_eps=1e-9, max_iter=500)
    check(s, tol)
