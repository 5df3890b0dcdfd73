"""The mixed form's field items: tile edges, masked partners with every scale,
walk parts and J chunks of every length the size rule picks.

Errors of the mixed field come from FP32 pair arithmetic (a few 1e-7 a pair,
1e-6 for the closest ones through the 1e-8 nm rounding of tile offsets), so the
dipoles have to agree within the mixed form's bound of 2e-5 relative RMS."""
import numpy as np
import pytest

from oracle import oracle as O
from tholedipoleplugin_b200 import systems as S
from tholedipoleplugin_b200.kernel import CudaCalcTholeDipoleForceKernel

from . import fixtures as F

pytestmark = pytest.mark.gpu


def rel_rms(a, b):
    return float(np.sqrt(np.mean((a - b) ** 2) / np.mean(b ** 2)))


@pytest.mark.parametrize("n", [4, 31, 32, 33, 63, 64, 65, 97, 200])
@pytest.mark.parametrize("method", [S.NO_CUTOFF, S.PME])
@pytest.mark.parametrize("polarization", [S.DIRECT, S.MUTUAL])
def test_tile_edges_and_partner_scales(n, method, polarization):
    # molecules of the random system overlap: small polarizabilities keep its dipole matrix positive definite
    s = F.small_random_system(n, seed=n, method=method, polarization=polarization, box=3.0)
    s = s.copy(polarizabilities=0.1 * s.polarizabilities, target_eps=1e-9, max_iter=2000)
    ref = O.compute(s.copy(target_eps=1e-12, max_iter=5000), "port").induced
    with CudaCalcTholeDipoleForceKernel(s, precision="mixed") as k:
        got = k.getInducedDipoles(s.positions)
    assert rel_rms(got, ref) < 2e-5


@pytest.mark.parametrize("n_side", [7, 11, 16, 20, 24])   # 8 and 1 parts of a walk, chunks of 1, 2, 4 and 8 J tiles
def test_chunk_lengths_match_plain_form(n_side):
    s = S.water_box(n_side, 0.3107 * n_side, seed=n_side, cutoff=0.8, target_eps=1e-8)
    for polarization in (S.DIRECT, S.MUTUAL):
        out = []
        for precision in ("mixed", "double"):
            with CudaCalcTholeDipoleForceKernel(s.copy(polarization=polarization), precision=precision) as k:
                out.append(k.getInducedDipoles(s.positions))
        assert rel_rms(*out) < 2e-5
