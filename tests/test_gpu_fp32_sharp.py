"""The FP32 step's launch forms against one another bit for bit, and its velocities and pressure
perturbations (not the pressure, which is 1 to four digits) against FP64."""
import numpy as np
import pytest

from mpdugks_gb300 import capi

pytestmark = pytest.mark.gpu

KW = dict(Mu0=0.02, M_Phi=0.05, W=4.0, Sigma=1e-3, RhoL=3.0, RhoV=1.0)


# undivided grids of the tile kernels (27x24, 420x421) and of the streaming kernel in segments of 5 rows
# and more, and the same grid as partitions, which stream in segments of other lengths
@pytest.mark.parametrize('model,walls', [('AC', True), ('HCZ', False), ('HCZ', True)])
@pytest.mark.parametrize('nx,ny', [(27, 24), (29, 1501), (420, 421), (450, 451), (741, 739)])
def test_tiles_and_segments_give_the_same_bits(nx, ny, model, walls):
    case = capi.make_case(model, 'fp32dev', **KW, **(dict(Gy=1e-5) if walls else {}))
    g, s = capi.GpuCase(case, nx, ny, walls), capi.Slabs(case, nx, ny, walls, 2)
    for x in (g, s):
        x.init('ac_rt', [0.5 * ny / nx, 0.1, 1e-3], seed=5)
        x.step(7)
    got = s.fields()
    s.close()
    for k in ('rho', 'u', 'v', 'phi', 'p'):
        assert np.array_equal(g.get(k), got[k]), k


# FP32 rounds the stored deviations, 1e-3 at most here, by 2^-24: a few 1e-10 after 40 steps against
# velocities of 1e-5 and more; a wrong flux at one seam would show at the velocities' own size
@pytest.mark.parametrize('kw,walls,nx,ny', [(dict(wall='NEE', Gy=1e-4), True, 61, 33), (dict(wall='NEE', Gy=1e-4), True, 741, 739),
                                             (dict(scheme='UW'), False, 61, 53), (dict(scheme='UW'), False, 607, 613),
                                             (dict(scheme='UW_LS'), False, 607, 613), (dict(scheme='UW_4P'), False, 91, 92)])
def test_velocities_and_pressures_close_to_fp64(kw, walls, nx, ny):
    out = []
    for prec in ('fp64', 'fp32dev'):
        g = capi.GpuCase(capi.make_case('HCZ', prec, **KW, **kw), nx, ny, walls)
        if walls:
            g.init('ac_rt', [0.5 * ny / nx, 0.05, 0.0])
        else:
            g.init('ac_drop_inside', [0.25 * min(nx, ny)])
        g.step(40)
        out.append({'u': g.get('u'), 'v': g.get('v'), 'p - 1': g.get('p') - 1.0})
    for k, ref in out[0].items():
        assert np.abs(ref).max() > 1e-6, k
        assert np.abs(out[1][k] - ref).max() <= 1e-4 * np.abs(ref).max(), k
