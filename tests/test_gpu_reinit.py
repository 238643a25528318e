"""A handle that is initialised again, after steps that leave its alternating copies either way round,
is the same as a new one."""
import numpy as np
import pytest

from mpdugks_gb300 import capi

pytestmark = pytest.mark.gpu

KW = dict(Mu0=0.02, M_Phi=0.05, W=4.0, Sigma=1e-3, RhoL=3.0, RhoV=1.0)
CASES = [('AC', 'ac_drop', [9.0], 'ac_rt', [0.5, 0.1, 1e-3], KW), ('HCZ', 'ac_rt', [0.5, 0.1, 1e-3], 'ac_drop_inside', [7.0], KW),
         ('PP9', 'scmp_drop', [], 'pp_noise', [0.2, 0.01], dict(Mu0=0.1)),
         ('PP16', 'pp_noise', [0.13, 0.01], 'scmp_drop', [], dict(Mu0=0.3, d2v16_c=0.5))]


def same(a, b, allen_cahn):
    for n in (0, 2):
        a.step(n)
        b.step(n)
        for w in ('f', 'h') if allen_cahn else ('f',):
            assert np.array_equal(a.dist(w), b.dist(w)), (n, w)
        for k in ('rho', 'u', 'v', 'p'):
            assert np.array_equal(a.get(k), b.get(k)), (n, k)
        assert a.reduce().steps == b.reduce().steps == n


@pytest.mark.parametrize('model,init,params,other,other_params,kw', CASES)
@pytest.mark.parametrize('precision,walls,passes', [('fp64', False, 3), ('fp64', True, 3), ('fp64fma', False, 3), ('fp32dev', False, 3),
                                                    ('fp32dev', True, 3), ('fp32dev', False, 1), ('fp64fused', True, 3)])
@pytest.mark.parametrize('before', [1, 4])
def test_initialised_again(model, init, params, other, other_params, kw, precision, walls, passes, before, monkeypatch):
    allen_cahn = model in ('AC', 'HCZ')
    if not allen_cahn and (walls or precision == 'fp64fused') or allen_cahn and passes == 1:
        pytest.skip('not a form of this model')
    monkeypatch.setenv('DUGKS_PP_PASSES', str(passes))
    nx, ny = 45, 37
    a, b = (capi.GpuCase(capi.make_case(model, precision, **kw), nx, ny, walls) for _ in range(2))
    a.init(other, other_params, seed=11)
    a.step(before)
    a.init(init, params, seed=12)
    b.init(init, params, seed=12)
    same(a, b, allen_cahn)


@pytest.mark.parametrize('model', ['AC', 'HCZ'])
@pytest.mark.parametrize('precision,walls', [('fp64fused', False), ('fp64fused', True), ('fp32dev', True), ('fp64', True)])
def test_an_upload_of_the_same_state_is_the_same(model, precision, walls):
    nx, ny = 33, 41
    ref = capi.GpuCase(capi.make_case(model, 'fp64', **KW), nx, ny, walls)
    a, b = (capi.GpuCase(capi.make_case(model, precision, **KW), nx, ny, walls) for _ in range(2))
    for g in (ref, a):
        g.init('ac_rt', [0.5, 0.1, 1e-3], seed=4)
    b.upload(ref.dist('f'), ref.dist('h'), np.stack([ref.get(k) for k in capi.FIELDS]))
    same(a, b, True)
