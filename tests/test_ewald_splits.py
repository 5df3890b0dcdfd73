"""The Ewald mode's mixed form against its plain form where the real-space walks
are split differently (32 ways for the smallest system, one for the largest) and
the last tile and the last group of five-lane atoms are ragged.

The mixed form's stated bounds: forces and dipoles 2e-5 relative RMS, energy 1e-6."""
import numpy as np
import pytest

from tholedipoleplugin_b200 import systems as S
from tholedipoleplugin_b200.kernel import CudaCalcTholeDipoleForceKernel

from .gpu_util import rel_err, rel_rms

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("polarization", [S.DIRECT, S.MUTUAL])
@pytest.mark.parametrize("n_side", [6, 7, 9, 13, 19])
def test_mixed_matches_plain(n_side, polarization):
    s = S.water_box(n_side, 0.3107 * n_side, seed=n_side, cutoff=0.8, target_eps=1e-8, polarization=polarization)
    out = []
    for precision in ("mixed", "double"):
        with CudaCalcTholeDipoleForceKernel(s, precision=precision, ewald=True) as k:
            e, f = k.execute(s.positions)
            out.append((e, f, k.getInducedDipoles()))
    (e, f, mu), (e0, f0, mu0) = out
    assert rel_err(e, e0) < 1e-6
    assert rel_rms(f, f0) < 2e-5
    assert rel_rms(mu, mu0) < 2e-5
