"""Checkpoints whose header is longer than this library's (earlier version 1 files carry the FP32
pseudopotential constants after the members that are read: 1400 or 456 bytes) and, for the FP32
upwind step, with another number of scratch planes after the state."""
import numpy as np
import pytest

from mpdugks_gb300 import capi

pytestmark = pytest.mark.gpu

BASE = dict(Mu0=0.01, M_Phi=0.05, W=4.0, Sigma=1e-3, RhoL=1.0, RhoV=0.1)
HEADER, ARENA_BYTES = 176, 136  # the members that are read; the offset of arena_bytes


def earlier(ck, constants, planes, floats):
    """The checkpoint as a library with `constants` more header bytes and `planes` more scratch
    planes of `floats` floats wrote it."""
    own = int(ck[12:16].view(np.uint32)[0])
    head, arena = ck[:HEADER].copy(), ck[own:]
    more = np.full(planes * floats * 4, 0xA5, np.uint8)
    head[12:16].view(np.uint32)[0] = HEADER + constants
    head[ARENA_BYTES:ARENA_BYTES + 8].view(np.uint64)[0] = arena.size + more.size
    return np.concatenate([head, np.full(constants, 0x5A, np.uint8), arena, more])


@pytest.mark.parametrize('model,prec,init,params,kw', [
    ('AC', 'fp64', 'ac_drop_inside', [5.0], BASE), ('HCZ', 'fp32dev', 'ac_drop_inside', [5.0], BASE),
    ('HCZ', 'fp64fused', 'ac_drop_inside', [5.0], BASE), ('PP16', 'fp32dev', 'scmp_drop', [], {}),
    ('PP9', 'fp64', 'scmp_drop', [], {}), ('HCZ', 'fp32dev', 'ac_drop_inside', [5.0], dict(BASE, scheme='UW'))])
@pytest.mark.parametrize('constants', [1400, 456])
def test_earlier_checkpoints_restore(model, prec, init, params, kw, constants):
    nx, ny = 20, 17
    a, b = (capi.GpuCase(capi.make_case(model, prec, **kw), nx, ny, False) for _ in range(2))
    a.init(init, params, seed=3)
    a.step(7)
    planes = 62 if 'scheme' in kw else 0
    ck = earlier(a.checkpoint(), constants, planes, -(-32 * ny * 4 // 256) * 64)
    b.restore(ck)
    for g in (a, b):
        g.step(5)
    for k in ('rho', 'u', 'v', 'p'):
        assert np.array_equal(a.get(k), b.get(k)), k
    assert np.array_equal(a.dist('f'), b.dist('f')) and a.reduce().steps == b.reduce().steps == 12
    for bad in (ck[:-1], ck[:HEADER + constants], ck[:HEADER]):
        with pytest.raises(capi.DugksError):
            b.restore(bad)
    with pytest.raises(capi.DugksError):
        capi.GpuCase(capi.make_case(model, prec, **kw), nx, ny + 1, False).restore(ck)
