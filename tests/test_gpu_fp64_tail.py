"""The exact FP64 step of a large grid whose phase field has its far tail (1e-80 and less, a cell
further at every step), where the integer-pipe products of its kernels do not apply."""
import time

import pytest

from mpdugks_gb300 import capi

pytestmark = pytest.mark.gpu

DROP = dict(Mu0=0.02, M_Phi=0.02, W=4.0, Sigma=1e-3, RhoL=1.0, RhoV=0.1)


def test_the_far_tail_costs_no_second_product():
    # a row of the tail takes the floating-point products, 11 % more time than the integer ones;
    # half the rows are in it: 6 % at most, where both kinds of product one after the other took 15
    first, late = (capi.GpuCase(capi.make_case('AC', 'fp64', **DROP), 512, 512, False) for _ in range(2))
    late.init('ac_drop_inside', [120.0])
    late.step(180)
    took = {first: 1.0, late: 1.0}
    for _ in range(6):  # in turn, so that both see the same clocks
        first.init('ac_drop_inside', [120.0])
        for g in (first, late):
            g.step(2)
            g.reduce()
            t = time.perf_counter()
            g.step(10)
            g.reduce()
            took[g] = min(took[g], time.perf_counter() - t)
    assert took[late] <= 1.09 * took[first]
