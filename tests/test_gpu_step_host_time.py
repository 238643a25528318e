"""What a step costs the calling thread does not grow with the grid's rows: the choice of the FP32
streaming step's segments, a search over the rows, is made once for a handle."""
import time

import pytest

from mpdugks_gb300 import capi

pytestmark = pytest.mark.gpu


def test_enqueueing_a_step_takes_microseconds():
    # a search over 100,000 lengths takes about 400 us; enqueueing a step 2 to 10
    g = capi.GpuCase(capi.make_case('HCZ', 'fp32dev', Mu0=0.1, M_Phi=0.1, W=4.0, Sigma=1e-3, RhoL=10.0, RhoV=1.0),
                     32, 100_000, False)
    g.init('ac_drop_inside', [8.0])
    g.step(1)
    best = 1.0
    for _ in range(5):
        g.reduce()  # waits for the steps before
        t = time.perf_counter()
        g.step(20)
        best = min(best, (time.perf_counter() - t) / 20)
    assert best < 100e-6
