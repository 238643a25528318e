"""What the pseudopotential steps give for a density that is not a number: the sign of p - rho RT
by the two comparisons of the reference, which are both false then."""
import numpy as np
import pytest

from mpdugks_gb300 import capi
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('model', ['PP9', 'PP16'])
def test_exact_sign_of_a_density_that_is_not_a_number(model):
    g, o = capi.GpuCase(capi.make_case(model, 'fp64'), 24, 20, False), Oracle(model, 24, 20, False, 'scmp_drop')
    g.init('scmp_drop', [])
    rho = g.get('rho')
    rho[9, 13] = np.nan
    g.set('rho', rho)
    o.set('rho', rho)
    for n in (1, 2):
        g.step(n)
        o.step(n)
        assert np.isnan(g.get('rho')).any() and not np.isnan(g.get('rho')).all()
        assert np.array_equal(g.get('scg'), o.get('scg'))
