"""The cluster batch's stored pair coefficients and lab-frame energy pass: a
cluster too large for the coefficient workspace, clusters of several rounds of
the thread split, pairs on the x axis, against one handle's evaluation.

Both run the same expressions in FP64 with sums of at most a few hundred terms
in another order and solves to 1e-11: 1e-9 of the largest force."""
import numpy as np
import pytest

from tholedipoleplugin_b200 import systems as S
from tholedipoleplugin_b200.batch import ClusterBatch
from tholedipoleplugin_b200.kernel import CudaCalcTholeDipoleForceKernel

pytestmark = pytest.mark.gpu


def chain(n, seed):
    """Atoms on the x axis (index order shuffled), one of them off it."""
    rng = np.random.default_rng(seed)
    pos = np.zeros((n, 3))
    pos[:, 0] = 0.3 * rng.permutation(n)
    pos[0, 1:] = 0.1
    axis = np.full((n, 4), -1, dtype=np.int32)
    axis[:, 0] = S.NOAXISTYPE
    return S.TholeSystem(positions=pos, charges=rng.normal(scale=0.4, size=n), dipoles=rng.normal(scale=0.01, size=(n, 3)),
                         polarizabilities=rng.uniform(0.3e-3, 1.5e-3, n), tholes=rng.uniform(0.3, 0.45, n), axis=axis,
                         cov12=[[] for _ in range(n)], cov13=[[] for _ in range(n)], target_eps=1e-11, max_iter=500)


CASES = {
    "small": lambda: [S.water_cluster(w, np.random.default_rng(w), target_eps=1e-11) for w in (1, 2, 5, 11, 21, 64)],
    "too_large_for_coefficients": lambda: [S.water_cluster(w, np.random.default_rng(w), target_eps=1e-11)
                                           for w in (100, 3)],
    "on_axis": lambda: [chain(n, n) for n in (2, 9, 40)],
}


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("polarization", [S.DIRECT, S.MUTUAL, S.EXTRAPOLATED])
def test_batch_equals_handles(name, polarization):
    clusters = [c.copy(polarization=polarization) for c in CASES[name]()]
    rng = np.random.default_rng(0)
    with ClusterBatch(clusters, precision="double") as b:
        e, f = b.compute()
        g = rng.normal(size=(b.n, 3))
        ge = rng.normal(size=len(clusters))
        # the reverse pass has no Extrapolated form and no room for 300 atoms
        grads = None if polarization == S.EXTRAPOLATED or name.startswith("too_large") else b.adjoint(g, ge)
        for k, c in enumerate(clusters):
            sl = b.cluster_slice(k)
            with CudaCalcTholeDipoleForceKernel(c, precision="double") as h:
                e0, f0 = h.execute(c.positions)
                g0 = h.adjoint(g[sl], float(ge[k]))
            assert abs(e[k] - e0) <= 1e-9 * max(abs(e0), np.abs(f0).max())
            assert np.abs(f[sl] - f0).max() <= 1e-9 * np.abs(f0).max()
            if grads is not None:
                for q in (slice(0, 1), slice(1, 2), slice(2, 3), slice(3, 6)):
                    assert np.abs(grads[sl, q] - g0[:, q]).max() <= 1e-8 * np.abs(g0[:, q]).max()


def test_adjoint_on_axis_against_differences():
    s = chain(9, 4)
    h = 1e-6
    with CudaCalcTholeDipoleForceKernel(s, precision="double") as k:
        k.execute(s.positions)
        g = k.adjoint(None, 1.0)

        def energy(**change):
            with CudaCalcTholeDipoleForceKernel(s.copy(**change), precision="double") as kk:
                return kk.execute(s.positions)[0]

        for i in (0, 3, 8):
            for col, name in ((0, "charges"), (1, "polarizabilities"), (2, "tholes")):
                base = getattr(s, name)
                step = np.zeros(s.n)
                step[i] = h * (abs(base[i]) + 1e-3)
                fd = (energy(**{name: base + step}) - energy(**{name: base - step})) / (2 * step[i])
                # central differences: h^2 truncation and 1e-11 / h of solver noise
                assert abs(fd - g[i, col]) <= 1e-4 * np.abs(g[:, col]).max()
