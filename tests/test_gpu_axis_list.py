"""The mixed form's list of pairs close to the x axis (16 an atom), where it is just full (a chain of 33
atoms has 528 pairs), just too short (34: 561 pairs, room for 544) and far too short: the same bits in every
run, and the plain form's results.

Tolerances are the mixed form's: forces 2e-5 relative RMS, energy 1e-6 |E| + 3e-7 sqrt(sum (q_i q_j /
r_ij)^2)."""
import numpy as np
import pytest

from tholedipoleplugin_b200 import _capi as A
from tholedipoleplugin_b200 import systems as S
from tholedipoleplugin_b200.kernel import CudaCalcTholeDipoleForceKernel

from .gpu_util import energy_rms_scale, rel_rms

pytestmark = pytest.mark.gpu


def chain(x, charges, tholes, dipoles, alpha):
    n = len(x)
    pos = np.zeros((n, 3))
    pos[:, 0] = x
    axis = np.full((n, 4), -1, dtype=np.int32)
    axis[:, 0] = S.NOAXISTYPE
    return S.TholeSystem(positions=pos, charges=charges, dipoles=dipoles, polarizabilities=alpha, tholes=tholes,
                         axis=axis, cov12=[[] for _ in range(n)], cov13=[[] for _ in range(n)],
                         polarization=S.DIRECT)


def random_chain(n):
    """Atoms 0.31 nm apart, shuffled within 32 of them (either orientation of a pair, compact tiles)."""
    rng = np.random.default_rng(n)
    x = np.concatenate([0.31 * (k + rng.permutation(min(32, n - k))) for k in range(0, n, 32)])
    return chain(x, rng.normal(scale=0.4, size=n), rng.uniform(0.3, 0.45, n), rng.normal(scale=0.01, size=(n, 3)),
                 rng.uniform(0.3e-3, 1.5e-3, n))


@pytest.mark.parametrize("n", [32, 33, 34, 362, 363, 400, 1000])
def test_chain_beyond_the_list(n):
    s = random_chain(n)
    runs = []
    for _ in range(3):
        with CudaCalcTholeDipoleForceKernel(s, precision="mixed", dd_force_r4=True) as k:
            runs += [k.execute(s.positions) for _ in range(2)]
    e, f = runs[0]
    for e1, f1 in runs[1:]:
        assert e1 == e and np.array_equal(f1, f)
    with CudaCalcTholeDipoleForceKernel(s, precision="double", dd_force_r4=True) as k:
        e0, f0 = k.execute(s.positions)
    assert rel_rms(f, f0) < 2e-5
    assert abs(e - e0) < 1e-6 * abs(e0) + 3e-7 * energy_rms_scale(s)


def test_sum_of_listed_pairs_beyond_the_range():
    """Every pair's share of the first atom's force is within the accumulator's limit (2^23 e^2/nm^2), their
    sum is beyond its range (2^31 at this size): an error, not a wrapped number."""
    n = 360
    x = np.concatenate([[0.0], np.linspace(1.0, 1.19, n - 1)])
    q = x ** 2
    q[0] = 6.6e6
    assert q[0] * 1.19 < 2 ** 23 and q[0] * (n - 1) > 2 ** 31 and (q[-1] / (x[-1] - x[-2])) ** 2 < 2 ** 23
    t = np.ones(n)   # the small charges' fields damp one another; the first atom's field is bare
    t[0] = 0.01
    s = chain(x, q, t, np.zeros((n, 3)), np.zeros(n))
    with CudaCalcTholeDipoleForceKernel(s, precision="mixed", dd_force_r4=True) as k:
        with pytest.raises(A.TdpError, match="accumulator range"):
            k.execute(s.positions)
    with CudaCalcTholeDipoleForceKernel(s, precision="double", dd_force_r4=True) as k:
        f0 = k.execute(s.positions)[1]
    assert abs(f0[0, 0]) > 2 ** 31
