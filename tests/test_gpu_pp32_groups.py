"""The FP32 pseudopotential step's tiles, by one and by two groups of threads, against the
single-pass form: the same arithmetic, so the same bits."""
import numpy as np
import pytest

from mpdugks_gb300 import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('model,kw', [('PP9', {}), ('PP16', dict(d2v16_c=0.5))])
@pytest.mark.parametrize('nx,ny', [(32, 8), (63, 9), (200, 161), (65, 1216), (33, 1825), (449, 257)])  # 1 .. 510 tiles
def test_tiles_equal_the_single_pass(model, kw, nx, ny, monkeypatch):
    out = []
    for passes in ('1', '3'):
        monkeypatch.setenv('DUGKS_PP_PASSES', passes)
        g = capi.GpuCase(capi.make_case(model, 'fp32dev', **kw), nx, ny, False)
        g.init('pp_noise', [0.13044, 0.01], seed=3)
        g.step(1)
        g.step(4)
        out.append([g.get(k) for k in ('rho', 'u', 'v', 'p', 'psi', 'fx', 'fy')] + list(g.dist('f')))
    for a, b in zip(*out):
        assert np.array_equal(a, b)
