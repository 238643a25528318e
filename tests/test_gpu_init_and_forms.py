"""The device-made initial states against the oracle's and against an upload of the same state, and
the exact FP64 step on grids that take each launch form: one-warp blocks, 32 x 8 blocks with the
integer-pipe products, and large grids of few columns."""
import numpy as np
import pytest

from mpdugks_gb300 import capi
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu

KW = dict(Mu0=0.02, M_Phi=0.05, W=4.0, Sigma=1e-3, RhoL=3.0, RhoV=1.0)
PP = dict(Tr=0.8, aCS=0.5, Tc_CS=0.0471625, Mu0=0.3, d2v16_c=0.5)


def gpu_case(model, precision, nx, ny, walls, init, params, **kw):
    g = capi.GpuCase(capi.make_case(model, precision, **kw), nx, ny, walls)
    g.init(init, params, seed=77)
    return g


@pytest.mark.parametrize('precision', ['fp32dev', 'fp64', 'fp64fma'])
@pytest.mark.parametrize('model,init,params,kw', [('AC', 'ac_drop', [9.0], KW), ('HCZ', 'ac_rt', [0.5, 0.1, 1e-3], KW),
                                                   ('PP9', 'scmp_drop', [], dict(Mu0=0.1)),
                                                   ('PP16', 'pp_noise', [0.13, 0.01], PP)])
@pytest.mark.parametrize('nx,ny', [(33, 17), (130, 131)])
def test_device_init_equals_upload_of_the_same_state(precision, model, init, params, kw, nx, ny):
    ref = gpu_case(model, 'fp64', nx, ny, False, init, params, **kw)
    f, aux = ref.dist('f'), np.stack([ref.get(k) for k in capi.FIELDS])
    h = ref.dist('h') if model in ('AC', 'HCZ') else None
    a = gpu_case(model, precision, nx, ny, False, init, params, **kw)
    b = capi.GpuCase(capi.make_case(model, precision, **kw), nx, ny, False)
    b.upload(f, h, aux)
    for n in (0, 2):
        a.step(n)
        b.step(n)
        assert np.array_equal(a.dist('f'), b.dist('f'))
        if h is not None:
            assert np.array_equal(a.dist('h'), b.dist('h'))
        for k in ('rho', 'u', 'v', 'p'):
            assert np.array_equal(a.get(k), b.get(k)), (n, k)


@pytest.mark.parametrize('model', ['AC', 'HCZ'])
@pytest.mark.parametrize('nx,ny,walls', [(31, 9, True), (479, 480, False), (480, 481, True), (33, 7100, True),
                                         (577, 401, False)])
def test_exact_step_in_every_launch_form_equals_the_oracle(model, nx, ny, walls):
    # a drop about (nx / 2, nx / 2); gravity between the walls
    kw = dict(KW, Gy=1e-4 if walls else 0.0)
    radius = 0.3 * min(nx, ny)
    g = gpu_case(model, 'fp64', nx, ny, walls, 'ac_drop_inside', [radius], **kw)
    o = Oracle(model, nx, ny, walls, 'ac_drop_inside', radius=radius, **kw)
    for n in (1, 4):
        g.step(n)
        o.step(n)
        for k in ('rho', 'u', 'v', 'phi', 'p'):
            assert np.array_equal(g.get(k), o.get(k)), (n, k)
