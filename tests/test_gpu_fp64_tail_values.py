"""The exact FP64 step against the oracle where the phase field beyond an interface has fallen to
1e-80 ... 1e-323."""
import numpy as np
import pytest

from mpdugks_gb300 import capi
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu

DROP = dict(Mu0=0.02, M_Phi=0.02, W=4.0, Sigma=1e-3, RhoL=1.0, RhoV=0.1)


@pytest.mark.parametrize('model', ['AC', 'HCZ'])
@pytest.mark.parametrize('nx,ny', [(480, 483), (200, 203)])
def test_a_drop_with_its_far_tail(model, nx, ny):
    # subnormal numbers round at 2^-1074, where a factor 1/2 taken out of a sum no longer commutes with
    # the rounding: values below 2^-1000 may differ by some units of that, all others not at all
    radius = 0.23 * nx
    g = capi.GpuCase(capi.make_case(model, 'fp64', **DROP), nx, ny, False)
    o = Oracle(model, nx, ny, False, 'ac_drop_inside', radius=radius, **DROP)
    g.init('ac_drop_inside', [radius])
    for n in (30, 90, 20):
        g.step(n)
        o.step(n)
        phi = np.abs(o.get('phi'))
        assert ((phi > 0) & (phi < 2.0 ** -255)).any()
        for k in ('rho', 'u', 'v', 'phi', 'p'):
            a, b = g.get(k), o.get(k)
            assert np.abs(a - b).max() <= 2.0 ** -1040, (n, k)
            assert np.array_equal(a[np.abs(b) > 2.0 ** -980], b[np.abs(b) > 2.0 ** -980]), (n, k)
