"""The FP32 streaming step in segments of few rows, and the grids on either side of the rule that
leaves a grid to the tile kernel, against FP64."""
import numpy as np
import pytest

from mpdugks_gb300 import capi

pytestmark = pytest.mark.gpu

KW = dict(Mu0=0.02, M_Phi=0.05, W=4.0, Sigma=1e-3, RhoL=3.0, RhoV=1.0)


@pytest.mark.parametrize('model,walls,kw', [('AC', False, {}), ('HCZ', True, dict(Gy=1e-5)),
                                            ('HCZ', True, dict(wall='NEE'))])
@pytest.mark.parametrize('nx,ny', [(27, 8), (29, 1501), (420, 421), (450, 451), (741, 739)])
def test_short_segments_close_to_fp64(nx, ny, model, walls, kw):
    # ten FP32 steps of a noisy interface round to a few 2^-24 each: within 2e-5
    out = {}
    for prec in ('fp32dev', 'fp64'):
        g = capi.GpuCase(capi.make_case(model, prec, **KW, **kw), nx, ny, walls)
        g.init('ac_rt', [0.5 * ny / nx, 0.1, 1e-3], seed=5)
        g.step(10)
        out[prec] = {k: g.get(k) for k in ('rho', 'p', 'phi')}
    for k, ref in out['fp64'].items():
        assert np.abs(out['fp32dev'][k] - ref).max() <= 2e-5 * np.abs(ref).max(), k
