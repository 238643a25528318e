"""The FP32 upwind step's tiles (30 x 6 cells, ragged last ones, both register budgets) against FP64."""
import numpy as np
import pytest

from mpdugks_gb300 import capi

pytestmark = pytest.mark.gpu

KW = dict(Mu0=0.02, M_Phi=0.05, W=4.0, Sigma=1e-3, RhoL=3.0, RhoV=1.0)


@pytest.mark.parametrize('scheme', ['UW', 'UW_LS', 'UW_4P'])
@pytest.mark.parametrize('model', ['AC', 'HCZ'])
@pytest.mark.parametrize('nx,ny', [(3, 7), (29, 5), (31, 13), (61, 12), (607, 613)])
def test_fp32_upwind_tiles_close_to_fp64(nx, ny, model, scheme):
    # from a noisy interface; ten FP32 steps round to a few 2^-24 each: within 2e-5
    out = {}
    for prec in ('fp32dev', 'fp64'):
        g = capi.GpuCase(capi.make_case(model, prec, scheme=scheme, **KW), nx, ny, False)
        g.init('ac_rt', [0.5 * ny / nx, 0.1, 1e-3], seed=5)
        g.step(10)
        out[prec] = {k: g.get(k) for k in ('rho', 'p', 'phi')}
    for k, ref in out['fp64'].items():
        assert np.abs(out['fp32dev'][k] - ref).max() <= 2e-5 * np.abs(ref).max(), k
