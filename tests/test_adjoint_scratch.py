"""The adjoint's pair pass: what its scratch may take (an atom's list row and its count, and 64 bytes for each
of at most nine J splits, fewer where the splits make eight rounds of 12 resident 32-atom blocks on 148 SMs),
the rows' length, and lists at and beyond it."""
import ctypes as C

import numpy as np
import pytest

from tholedipoleplugin_b200 import _capi as A
from tholedipoleplugin_b200 import build as B
from tholedipoleplugin_b200 import systems as S
from tholedipoleplugin_b200.kernel import CudaCalcTholeDipoleForceKernel


@pytest.fixture(scope="module")
def lib():
    B.build()
    lib = A.lib()
    lib._ZN3tdp20adjoint_pair_scratchEii.argtypes = [C.c_int, C.c_int]   # tdp::adjoint_pair_scratch, in doubles
    lib._ZN3tdp20adjoint_pair_scratchEii.restype = C.c_size_t
    lib._ZN3tdp16adjoint_list_capEid.argtypes = [C.c_int, C.c_double]    # tdp::adjoint_list_cap
    return lib


@pytest.mark.parametrize("n", [1, 32, 33, 192, 1029, 6303, 6336, 12288, 12608, 12640, 28384, 28448, 50528, 50560, 98304,
                               200000, 227328, 227360, 1000000])
def test_pair_scratch(lib, n):
    cap = lib._ZN3tdp16adjoint_list_capEid(n, 190.0)
    assert cap == 256   # liquid water
    splits = min(9, max(1, 8 * 12 * 148 // -(-n // 32)))
    got = 8 * lib._ZN3tdp20adjoint_pair_scratchEii(n, cap)
    assert n * (4 * (cap + 1) + 64) <= got <= n * (4 * (cap + 1) + 64 * splits) + 8


@pytest.mark.parametrize("n,expected,cap", [(5, 5.0, 256), (300, 300.0, 320), (258, 300.0, 320), (10000, 150.0, 256), (10000, 385.0, 512),
                                            (10000, 5000.0, 2048), (10000, 10000.0, 2048)])
def test_list_cap(lib, n, expected, cap):
    assert lib._ZN3tdp16adjoint_list_capEid(n, expected) == cap


def dense_system(n):
    """Every pair within the damping range (3.7 nm at Thole factors of 1, jittered against ties)."""
    rng = np.random.default_rng(n)
    m = int(np.ceil(n ** (1 / 3)))
    pos = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[rng.permutation(m ** 3)[:n]] * 0.3
    axis = np.full((n, 4), -1, dtype=np.int32)
    axis[:, 0] = S.NOAXISTYPE
    cov = [[i + 1] if i % 3 == 0 and i + 1 < n else [] for i in range(n)]
    return S.TholeSystem(positions=pos + rng.uniform(-0.05, 0.05, (n, 3)), charges=rng.normal(scale=0.4, size=n),
                         dipoles=rng.normal(scale=0.01, size=(n, 3)), polarizabilities=rng.uniform(0.3e-3, 1.0e-3, n),
                         tholes=rng.uniform(0.95, 1.05, n), axis=axis, cov12=cov, cov13=[[] for _ in range(n)],
                         target_eps=1e-13, max_iter=500)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [192, 257, 258, 300])   # 191 to 299 damped partners an atom
def test_full_lists(n):
    """Central differences of the FP64 form's own loss; a step of 1e-5 leaves 1e-10 of curvature and 1e-11 of
    cancellation, against the 1e-6 asked."""
    s = dense_system(n)
    rng = np.random.default_rng(1)
    g = rng.normal(size=(n, 3))
    with CudaCalcTholeDipoleForceKernel(s, precision="double") as k:

        def loss(q, a, t):
            k.copyParametersToContext(s.copy(charges=q, polarizabilities=a, tholes=t))
            e, f = k.execute(s.positions)
            return 0.7 * e + float((g * f).sum())

        p = [s.charges, s.polarizabilities, s.tholes]
        loss(*p)
        grad = k.adjoint(g, 0.7)
        for c in range(3):
            for i in (0, n // 2, n - 1):
                h = 1e-5 * abs(p[c][i])
                v = []
                for sign in (1.0, -1.0):
                    q = [x.copy() for x in p]
                    q[c][i] += sign * h
                    v.append(loss(*q))
                assert abs(grad[i, c] - (v[0] - v[1]) / (2 * h)) < 1e-6 * np.abs(grad[:, c]).max(), (c, i)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["mixed", "double"])
@pytest.mark.parametrize("n_side", [6, 11])
def test_same_bits_in_every_run(n_side, precision):
    """The splits of an atom share its list row."""
    s = S.water_box(n_side, 0.3107 * n_side, seed=2, cutoff=0.8, target_eps=1e-7)
    g = np.random.default_rng(1).normal(size=(s.n, 3))
    runs = []
    for _ in range(2):
        with CudaCalcTholeDipoleForceKernel(s, precision=precision) as k:
            k.execute(s.positions)
            runs += [k.adjoint(g, 0.3) for _ in range(3)]
    for r in runs[1:]:
        assert np.array_equal(r, runs[0])


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["mixed", "double"])
def test_rows_follow_the_thole_factors(precision):
    """After an adjoint at factors that damp next to nothing, one at factors that damp every pair is the one
    of a new handle: its rows hold the 299 partners (shorter ones are scanned, in another order)."""
    s = dense_system(300)
    g = np.random.default_rng(1).normal(size=(s.n, 3))
    out = []
    for first in (0.05, None):
        with CudaCalcTholeDipoleForceKernel(s, precision=precision) as k:
            if first is not None:
                k.copyParametersToContext(s.copy(tholes=first * s.tholes, polarizabilities=0.1 * s.polarizabilities))
                k.execute(s.positions)
                k.adjoint(g, 0.7)
                k.copyParametersToContext(s)
            k.execute(s.positions)
            out.append(k.adjoint(g, 0.7))
    assert np.array_equal(*out)
