"""The FP32 D2V16 step is as near to FP64 as it was with the inverse moment matrix's entries rounded
one by one: the relative error of u, of a growing density noise, averaged over three seeds."""
import numpy as np
import pytest

from mpdugks_gb300 import capi

pytestmark = pytest.mark.gpu

EOS = dict(aCS=0.5, Tc_CS=0.3773 * 0.5 / 4.0, d2v16_c=0.5, Mu0=0.3, Tr=0.75)


# the matrix form's errors of these runs: 4.589e-6 and 1.299e-5
@pytest.mark.parametrize('nx,ny,steps,bound', [(300, 280, 50, 4.6e-6), (64, 96, 200, 1.31e-5)])
def test_velocity_error_against_fp64(nx, ny, steps, bound):
    errors = []
    for seed in (2, 3, 4):
        u = []
        for prec in ('fp64', 'fp32dev'):
            g = capi.GpuCase(capi.make_case('PP16', prec, **EOS), nx, ny, False)
            g.init('pp_noise', [0.13044, 0.01], seed=seed)
            g.step(steps)
            u.append(g.get('u'))
        errors.append(np.linalg.norm(u[1] - u[0]) / np.linalg.norm(u[0]))
    assert np.mean(errors) <= bound
