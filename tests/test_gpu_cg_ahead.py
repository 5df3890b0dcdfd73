"""An iteration queued before the host has seen that the solve has stopped: its matvec does nothing.

A matvec of this size walks 528,906 pairs (10 us or more); a kernel that returns at once takes about 2 us."""
import numpy as np
import pytest
import torch
from torch.profiler import ProfilerActivity, profile

from tholedipoleplugin_b200 import systems as S
from tholedipoleplugin_b200.kernel import CudaCalcTholeDipoleForceKernel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,kernel", [("mixed", "k_field_items<1"), ("double", "k_field_bands<1")])
def test_matvec_after_the_last_iteration(precision, kernel):
    s = S.water_box(7, 0.3107 * 7, seed=7, cutoff=0.9, target_eps=1e-7)
    with CudaCalcTholeDipoleForceKernel(s, precision=precision) as k:
        k.getInducedDipoles(s.positions)   # sorted, loaded
        with profile(activities=[ProfilerActivity.CUDA]) as p:
            k.getInducedDipoles(s.positions)
            torch.cuda.synchronize()
        steps = k.solverStats()["iterations"]
    us = [e.device_time for e in p.events() if kernel in e.name.replace("(int)", "")]
    if not us:
        pytest.skip("the profiler records no kernels here")
    # one walk a step, one queued ahead of the stop, perhaps one for the true residual
    assert steps + 1 <= len(us) <= steps + 3
    assert sum(t > 0.5 * np.median(us) for t in us) <= len(us) - 1
    assert min(us) < 0.35 * np.median(us)
