"""The workloads this framework's speed is judged by.

One pass is what a solver loop does between two looks at its case: a number of time
steps, the density and phase sums that the residual check reads, and a download of the
macroscopic fields.  The sizes and constants are those of the benchmark's configurations
(the 512x2048 and large Rayleigh-Taylor boxes, the 128x128 Allen-Cahn drop, the
1024x1024 D2V16 separation, the serving stream) and of the tests.

FP64 results are kept as the doubles the library hands out; FP32 storage holds 32-bit
values, and its fields are kept as float32.
"""
import ctypes
import math

import numpy as np
import torch

from mpdugks_gb300 import capi

NAMES = ('rho', 'u', 'v', 'phi', 'p')

# constants of the drops, the Rayleigh-Taylor boxes and the pseudopotential cases
AC_DROP = dict(Mu0=0.02, M_Phi=0.02, W=4.0, Sigma=1e-3, RhoL=1.0, RhoV=0.1)
HCZ_DROP = dict(Mu0=0.1, M_Phi=0.1, W=4.0, Sigma=1e-3, RhoL=10.0, RhoV=1.0)
PP_EOS = dict(aCS=0.5, Tc_CS=0.3773 * 0.5 / 4.0, d2v16_c=0.5, Mu0=0.3)
RHO_C = 0.13044


def listed():
    return [
        # the reference's own small test case, FP64: launches and latency
        dict(name='ac_drop_32x24_fp64', kind='run', model='AC', precision='fp64', nx=32, ny=24, steps=50),
        # the reference's default case, 128x128 Allen-Cahn drop, in the default precision
        dict(name='ac_drop_128x128_fp64', kind='run', model='AC', precision='fp64', nx=128, ny=128, steps=50),
        # the Rayleigh-Taylor configuration, walls and gravity, in the default precision
        dict(name='rt_512x2048_fp64', setup='rt', kind='run', model='HCZ', precision='fp64', nx=512, ny=2048, steps=5),
        # an odd periodic box with FMA contraction
        dict(name='hcz_drop_333x257_fp64fma', kind='run', model='HCZ', precision='fp64fma', nx=333, ny=257, steps=40),
        # a small case in FP32 storage, stepped on its own
        dict(name='hcz_drop_128x128_fp32', kind='run', model='HCZ', precision='fp32dev', nx=128, ny=128, steps=200),
        # end to end from a host state: upload, run, read back
        dict(name='rt_512x2048_fp32_e2e', setup='rt', kind='e2e', model='HCZ', precision='fp32dev', nx=512, ny=2048,
             steps=200),
        # the large Rayleigh-Taylor box, state far beyond L2
        dict(name='rt_3072x3072_fp32', setup='rt', kind='run', model='HCZ', precision='fp32dev', nx=3072, ny=3072,
             steps=100),
        # the reference's other flux scheme
        dict(name='uw_drop_512x512_fp32', kind='run', model='HCZ', precision='fp32dev', nx=512, ny=512, steps=100,
             scheme='UW'),
        # phase separation with the D2V16 model, production precision and the exact one
        dict(name='pp16_1024x1024_fp32', kind='run', model='PP16', precision='fp32dev', nx=1024, ny=1024, steps=50),
        dict(name='pp16_256x256_fp64', kind='run', model='PP16', precision='fp64', nx=256, ny=256, steps=20),
        # a pseudopotential drop on an odd grid
        dict(name='pp9_drop_150x133_fp32', kind='run', model='PP9', precision='fp32dev', nx=150, ny=133, steps=200),
        # the request loop: a mix of small cases submitted at once
        dict(name='serve_24', kind='serve', cases=24, stream=1, steps=300),
    ]


def log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['fp64', 'fp64', 'fp64fma', 'fp32', 'fp32', 'fp32', 'e2e', 'uw', 'pp32', 'pp32', 'pp64', 'serve'])
    if kind == 'serve':
        return dict(kind='serve', cases=rng.randint(4, 32), stream=rng.randint(2, 1 << 20), steps=300)
    model = rng.choice(['AC', 'HCZ', 'HCZ'])
    if kind in ('fp64', 'fp64fma'):
        nx, ny, budget, precision = log_int(rng, 24, 700), log_int(rng, 24, 1500), 4e6, kind
    elif kind in ('fp32', 'e2e'):
        nx, ny, budget, precision = log_int(rng, 32, 3000), log_int(rng, 32, 3000), 8e8, 'fp32dev'
    elif kind == 'uw':
        nx, ny, budget, precision = log_int(rng, 32, 1200), log_int(rng, 32, 1200), 4e7, 'fp32dev'
    else:
        model = rng.choice(['PP9', 'PP16', 'PP16'])
        nx, ny, budget, precision = log_int(rng, 32, 1100), log_int(rng, 32, 1100), 4e7, 'fp32dev'
        if kind == 'pp64':
            nx, ny, budget = log_int(rng, 24, 400), log_int(rng, 24, 400), 1.5e6
            precision = rng.choice(['fp64', 'fp64fma'])
    if kind == 'e2e':
        nx, ny = min(nx, 1600), min(ny, 1600)
    rt = model == 'HCZ' and kind != 'uw' and rng.random() < 0.6
    if not rt and model != 'PP16':  # a drop sits at (nx / 2, nx / 2)
        ny = max(24, int(nx * rng.uniform(0.75, 1.3)))
    steps = max(4, min(200, int(budget / (nx * ny))))
    out = dict(kind='e2e' if kind == 'e2e' else 'run', model=model, precision=precision, nx=nx, ny=ny, steps=steps)
    if rt:
        out['setup'] = 'rt'
    if kind == 'uw':
        out['scheme'] = rng.choice(['UW', 'UW_LS', 'UW_4P'])
    return out


# ---------------------------------------------------------------- the cases' parameters

def physics(case, seed):
    """(constants, y walls, initialisation, its parameters) of one case; the seed places the drop,
    the interface or the noise."""
    g = np.random.default_rng([seed, case['nx'], case['ny']])
    n = min(case['nx'], case['ny'])
    if case['model'] == 'PP16':
        return dict(PP_EOS, Tr=0.7 + 0.1 * g.random()), False, 'pp_noise', [RHO_C, 0.01]
    if case['model'] == 'PP9':
        return dict(Mu0=0.1, Tr=0.85), False, 'scmp_drop', [2.4806e-1, 4.5435e-2, n * (0.2 + 0.1 * g.random())]
    if case.get('setup') == 'rt':
        # Rayleigh-Taylor between walls: heavy fluid above a cosine interface, gravity
        nx = float(case['nx'])
        kw = dict(Mu0=max(0.01, 0.04 * nx / 10000.0), M_Phi=0.02, W=4.0, Sigma=5e-5, RhoL=3.0, RhoV=1.0,
                  Gy=0.04 ** 2 / nx)
        return kw, True, 'ac_rt', [0.5 * case['ny'] / nx, (0.03 + 0.04 * g.random()) * case['ny'] / nx, 1e-4]
    kw = HCZ_DROP if case['model'] == 'HCZ' else AC_DROP
    return kw, False, 'ac_drop_inside', [n * (0.2 + 0.1 * g.random())]


def serving_requests(case, seed):
    """The cases of one serving pass: sizes from the stream's lognormal distribution (median 256),
    70% Allen-Cahn drops and bubbles, 30% D2V16 separations.  The sizes belong to the case, the
    physics to the seed."""
    size, phys = np.random.default_rng(case['stream']), np.random.default_rng([seed, case['stream']])
    out = []
    for _ in range(case['cases']):
        n = int(np.clip(round(256 * math.exp(size.normal(0.0, math.log(4.0) / 2))), 64, 512))
        if size.random() < 0.7:
            kw = dict(Mu0=0.02, M_Phi=0.02, W=4.0, Sigma=float(phys.uniform(1e-4, 1e-2)), RhoL=1.0,
                      RhoV=float(1.0 / phys.uniform(2.0, 100.0)))
            out.append(dict(model='AC', n=n, kw=kw, init='ac_drop' if phys.random() < 0.5 else 'ac_drop_inside',
                            params=[n * float(phys.uniform(0.18, 0.25))]))
        else:
            out.append(dict(model='PP16', n=n, kw=dict(PP_EOS, Tr=float(phys.uniform(0.7, 0.85))), init='pp_noise',
                            params=[RHO_C, 0.01]))
    return out


# ---------------------------------------------------------------- what a program keeps and runs

class Solve:
    """A resident case with the host buffers its fields are read into."""

    def __init__(self, case, seed):
        kw, walls, init, params = physics(case, seed)
        nx, ny = case['nx'], case['ny']
        cs = capi.make_case(case['model'], case['precision'], scheme=case.get('scheme', 'CD'), **kw)
        self.gpu = capi.GpuCase(cs, nx, ny, walls)
        self.steps = case['steps']
        self.host = None
        if case['kind'] == 'e2e':  # the caller's own state, in pinned memory
            st = initial(case, seed)
            aux = torch.zeros(len(capi.FIELDS), ny, nx, dtype=torch.float64, device='cuda')
            for k, name in enumerate(capi.FIELDS):
                if name in st:
                    aux[k] = st[name]
            self.host = [torch.stack(st[k]).cpu().pin_memory().numpy() for k in ('f', 'h')] + \
                        [aux.cpu().pin_memory().numpy()]
        else:
            self.gpu.init(init, params, seed=seed % (1 << 32) + 1)
        self.fields = torch.empty(len(NAMES), ny, nx, dtype=torch.float64, pin_memory=True)
        self.ptrs = [ctypes.c_void_p(t.data_ptr()) for t in self.fields]
        self.kept = torch.zeros(len(NAMES), ny, nx, dtype=torch.float32) if case['precision'] == 'fp32dev' else None
        self.has_phi = case['model'] in ('AC', 'HCZ')

    def run(self):
        if self.host is not None:
            self.gpu.upload(*self.host)
        self.gpu.step(self.steps)
        sums = self.gpu.reduce()
        rc = self.gpu.lib.dugks_gpu_download(self.gpu.h, *self.ptrs)
        if rc != capi.DUGKS_OK:
            raise RuntimeError('download failed: %s' % capi.STATUS_NAMES[rc])
        out = self.fields if self.kept is None else self.kept.copy_(self.fields)
        got = {k: out[i] for i, k in enumerate(NAMES) if self.has_phi or k != 'phi'}
        got['sum_rho'] = float(sums.sum_rho)
        if self.has_phi:
            got['sum_phi'] = float(sums.sum_phi)
        return got


class Serve:
    """A server and the requests one pass sends to it."""

    def __init__(self, case, seed):
        self.server = capi.Server(max_bytes=8 << 30)
        self.seed = seed % (1 << 32) + 1
        self.requests = [(capi.make_case(r['model'], 'fp32dev', **r['kw']), r) for r in serving_requests(case, seed)]
        self.steps = case['steps']

    def run(self):
        srv = self.server
        ids = [srv.submit(cs, r['n'], r['n'], False, r['init'], r['params'], seed=self.seed + k, nsteps=self.steps)
               for k, (cs, r) in enumerate(self.requests)]
        out = []
        for cid, (_, r) in zip(ids, self.requests):
            st = srv.wait(cid)
            if capi.SRV_STATES[st.state] != 'done':
                raise RuntimeError('a served case ended %s' % capi.SRV_STATES[st.state])
            res = srv.result(cid)
            srv.release(cid)
            names = ('rho', 'phi') if r['model'] == 'AC' else ('rho', 'u')
            out.append([res[k].astype(np.float32) for k in names])
        return out


def prepare(case, seed):
    return Serve(case, seed) if case['kind'] == 'serve' else Solve(case, seed)


def run(state):
    return state.run()


# operations of one cell-update: reconstruction, moments, equilibria and sources of two faces
# and the cell, and the update, each shared sub-expression counted once
FLOPS = {'AC': 600, 'HCZ': 1100, 'PP9': 900, 'PP16': 1800}


def work(case):
    if case['kind'] == 'serve':
        b = f = 0
        for r in serving_requests(case, 0):
            w = work(dict(kind='run', model=r['model'], precision='fp32dev', nx=r['n'], ny=r['n'], steps=case['steps']))
            b, f = b + w['bytes'], f + w['flops']
        return {'bytes': b, 'flops': f}
    cells = case['nx'] * case['ny']
    # the compulsory state, read and written once a step: 18 distributions and the previous
    # phi u (two components), or the 9 / 16 distributions and psi, its sign of the pseudopotential models
    planes = {'AC': 20, 'HCZ': 20, 'PP9': 11, 'PP16': 18}[case['model']]
    size = 4 if case['precision'] == 'fp32dev' else 8
    moved = 2 * planes * size * cells * case['steps']
    fields = 5 * 8 * cells
    up = (9 + 9 + len(capi.FIELDS)) * 8 * cells if case['kind'] == 'e2e' else 0
    return {'bytes': moved + fields + up, 'flops': FLOPS[case['model']] * cells * case['steps']}


# ---------------------------------------------------------------- the same step in plain torch, 64 bits

XU9, XV9 = [0, 1, 1, 0, -1, -1, -1, 0, 1], [0, 0, 1, 1, 1, 0, -1, -1, -1]
W9 = [4 / 9] + [1 / 9, 1 / 36] * 4
BB9 = [0, 5, 6, 7, 8, 1, 2, 3, 4]
XU16 = [1, 0, -1, 0, 1, -1, -1, 1, 2, 0, -2, 0, 2, -2, -2, 2]
XV16 = [0, 1, 0, -1, 1, 1, -1, -1, 0, 2, 0, -2, 2, 2, -2, -2]
RT = 1.0 / 3.0


def lcg_noise(seed, n):
    """n values in [0, 1) of the initialisations' 64-bit generator x -> a x + c."""
    a, c = np.array([6364136223846793005], np.uint64), np.array([1442695040888963407], np.uint64)
    while a.size < n:  # the k-th value is A_k seed + C_k; the second half follows from the first
        c = np.concatenate([c, a * c[-1] + c])
        a = np.concatenate([a, a * a[-1]])
    x = a[:n] * np.uint64(seed) + c[:n]
    return (x >> np.uint64(11)).astype(np.float64) / 9007199254740992.0


def initial(case, seed):
    """The initial state as torch planes: f, h and the macroscopic fields."""
    kw, walls, init, params = physics(case, seed)
    return initial_state(case['model'], kw, init, params, seed % (1 << 32) + 1, case['nx'], case['ny'])


def initial_state(model, kw, init, params, seed, nx, ny):
    x = torch.arange(nx, dtype=torch.float64, device='cuda') + 0.5
    y = (torch.arange(ny, dtype=torch.float64, device='cuda') + 0.5)[:, None]
    zero = torch.zeros(ny, nx, dtype=torch.float64, device='cuda')
    r = torch.sqrt((x - 0.5 * nx) ** 2 + (y - 0.5 * nx) ** 2)
    if init in ('ac_rt', 'pp_noise'):
        noise = torch.from_numpy(lcg_noise(seed, nx * ny)).cuda().reshape(ny, nx) * 2.0 - 1.0
    st = {'u': zero, 'v': zero}
    if model in ('PP9', 'PP16'):
        if init == 'pp_noise':
            rho = params[0] * (1.0 + params[1] * noise)
        else:
            rl, rv, rad = params
            rho = 0.5 * (rl + rv) - 0.5 * (rv - rl) * torch.tanh(2 * (r - rad) / 5.0)
        st.update(rho=rho, p=rho * RT, f=pp_equilibrium(model, kw, rho, zero, zero))
        return st
    w = kw['W']
    if init == 'ac_rt':
        yi = nx * (params[0] + params[1] * torch.cos(2.0 * math.pi * x / nx))
        phi = 0.5 + 0.5 * torch.tanh((y - yi) * 2 / w) + params[2] * noise
    else:
        d = params[0] - r if init == 'ac_drop_inside' else r - params[0]
        phi = 0.5 + 0.5 * torch.tanh(d * 2 / w)
    rho = (kw['RhoL'] - kw['RhoV']) * phi + kw['RhoV']
    one = torch.ones_like(phi)
    st.update(phi=phi, rho=rho, p=one, tauf=kw['Mu0'] / (rho * RT), h=[wq * phi for wq in W9],
              f=[wq * one if model == 'HCZ' else (wq - (q == 0)) / RT * one for q, wq in enumerate(W9)])
    return st


def wrap(a, walls):
    """a with one row more on each side: periodic, or extrapolated beyond a wall."""
    lo, hi = (2 * a[:1] - a[1:2], 2 * a[-1:] - a[-2:-1]) if walls else (a[-1:], a[:1])
    return torch.cat([lo, a, hi])


def east(a):
    return torch.roll(a, -1, 1)


def west(a):
    return torch.roll(a, 1, 1)


def iso_gradient(e):
    """The 8-neighbour gradient of a field given with its extra rows."""
    n, s, c = e[2:], e[:-2], e[1:-1]
    gx = 4 * (east(c) - west(c)) + (east(n) - west(n) + east(s) - west(s))
    gy = 4 * (n - s) + (east(n) - east(s) + west(n) - west(s))
    return gx / 12, gy / 12


def cell_gradient(e, scheme):
    if scheme == 'UW':
        return iso_gradient(e)
    return (east(e) - west(e))[1:-1] / 2, (e[2:] - e[:-2]) / 2  # least squares and 4 points agree on unit cells


def face_value(a, walls, xu, xv, hdt, along_x, scheme):
    """The half-step value of one distribution on the west faces (ny rows) or the south faces
    (ny + 1 rows)."""
    e = wrap(a, walls)
    if scheme == 'CD':
        if along_x:
            t = e[2:] - e[:-2]
            o, n, gx, gy = west(a), a, a - west(a), 0.25 * (t + west(t))
        else:
            t = east(e) - west(e)
            o, n, gx, gy = e[:-1], e[1:], 0.25 * (t[1:] + t[:-1]), e[1:] - e[:-1]
        return 0.5 * (o + n) - hdt * (gx * xu + gy * xv)
    gx, gy = cell_gradient(e, scheme)
    if along_x:
        so, sn, s = (west(a), west(gx), west(gy)), (a, gx, gy), xu
        fo, fn = (0.5 - hdt * xu, -hdt * xv), (-0.5 - hdt * xu, -hdt * xv)
    else:
        ge = [wrap(k, False) for k in (gx, gy)]
        so, sn, s = (e[:-1], ge[0][:-1], ge[1][:-1]), (e[1:], ge[0][1:], ge[1][1:]), xv
        fo, fn = (-hdt * xu, 0.5 - hdt * xv), (-hdt * xu, -0.5 - hdt * xv)
    vo, vn = (b + dx * g1 + dy * g2 for (b, g1, g2), (dx, dy) in ((so, fo), (sn, fn)))
    return vo if s > 0 else vn if s < 0 else 0.5 * (vo + vn)


def ac_equilibrium(model, rho, u, v, phi, p, src, grho, force):
    """(f eq, f source, h eq, h source) of every direction."""
    out = []
    uu = (u * u + v * v) / (2 * RT)
    for q in range(9):
        xu, xv, w = XU9[q], XV9[q], W9[q]
        if model == 'AC':
            fe = w * p / RT - (p / RT if q == 0 else 0)
            out.append((fe, w * (xu * force[0] + xv * force[1]) / RT, w * phi, w * (xu * src[0] + xv * src[1])))
            continue
        u1 = (xu * u + xv * v) / RT
        g = u1 + 0.5 * u1 * u1 - uu
        cu, cv = xu - u, xv - v
        so = w * ((1 + g) * (cu * force[0] + cv * force[1]) + g * RT * (cu * grho[0] + cv * grho[1]))
        out.append((w * (p + rho * g * RT), so, w * (1 + u1) * phi, w * (xu * src[0] + xv * src[1])))
    return out


def ac_run(model, kw, walls, scheme, st, steps):
    """Allen-Cahn models: `steps` steps from the state `st`."""
    dt, a_phi, nu = 0.5, kw['RhoL'] - kw['RhoV'], kw['Mu0']
    hdt, tau0, tau_h = 0.5 * dt, nu / RT, kw['M_Phi'] / RT
    beta, kappa, gy = 12.0 * kw['Sigma'] / kw['W'], 1.5 * kw['Sigma'] * kw['W'], kw.get('Gy', 0.0)
    f, h, rho, u, v, phi, p, tau = [st[k] for k in ('f', 'h', 'rho', 'u', 'v', 'phi', 'p', 'tauf')]
    zero = torch.zeros_like(rho)
    src, grho, force, old = [zero, zero], [zero, zero], [zero, zero], (zero, zero)
    for _ in range(steps):
        a, ah = (2 * tau - hdt) / (2 * tau + dt), (2 * tau_h - hdt) / (2 * tau_h + dt)
        eqs = ac_equilibrium(model, rho, u, v, phi, p, src, grho, force)
        bf = [a * f[q] + (1 - a) * (fe + tau * fs) for q, (fe, fs, _, _) in enumerate(eqs)]
        bh = [ah * h[q] + (1 - ah) * (he + tau_h * hs) for q, (_, _, he, hs) in enumerate(eqs)]
        flux = []
        for along_x in (True, False):
            xi = XU9 if along_x else XV9
            ff, fh = ([face_value(b[q], walls, XU9[q], XV9[q], hdt, along_x, scheme) for q in range(9)]
                      for b in (bf, bh))
            ext = [wrap(k, walls) for k in src + grho + force]
            sx, sy, rx, ry, fx, fy = [0.5 * (west(e) + e)[1:-1] if along_x else 0.5 * (e[:-1] + e[1:]) for e in ext]
            ph = sum(fh)
            rh = a_phi * ph + kw['RhoV']
            if model == 'AC':
                uu = vv = torch.zeros_like(ph)
                pp = (sum(ff) - ff[0]) * RT * 9 / 5
            else:
                uu = (sum(x * b for x, b in zip(XU9, ff)) + 0.5 * hdt * fx) / (rh * RT)
                vv = (sum(x * b for x, b in zip(XV9, ff)) + 0.5 * hdt * fy) / (rh * RT)
                pp = sum(ff) + 0.5 * hdt * RT * (rx * uu + ry * vv)
            b, bhh = 2 * tau0 / (2 * tau0 + hdt), 2 * tau_h / (2 * tau_h + hdt)
            eqs = ac_equilibrium(model, rh, uu, vv, ph, pp, (sx, sy), (rx, ry), (fx, fy))
            ff = [b * ff[q] + (1 - b) * (fe + tau0 * fs) for q, (fe, fs, _, _) in enumerate(eqs)]
            fh = [bhh * fh[q] + (1 - bhh) * (he + tau_h * hs) for q, (_, _, he, hs) in enumerate(eqs)]
            if walls and not along_x:  # bounce-back of the directions that enter the fluid
                for k in (ff, fh):
                    was = [b.clone() for b in k]
                    for q in range(9):
                        row = 0 if XV9[q] > 0 else -1
                        if XV9[q]:
                            k[q][row] = was[BB9[q]][row]
            flux.append([[x * b for x, b in zip(xi, k)] for k in (ff, fh)])

        def net(which, q):
            ax, ay = flux[0][which][q], flux[1][which][q]
            return dt * (ax - east(ax) + ay[:-1] - ay[1:])
        f = [4 / 3 * bf[q] - f[q] / 3 + net(0, q) for q in range(9)]
        h = [4 / 3 * bh[q] - h[q] / 3 + net(1, q) for q in range(9)]
        was = phi
        phi = sum(h)
        rho = a_phi * phi + kw['RhoV']
        tau = torch.full_like(rho, tau0)
        if model == 'AC':
            p = (sum(f) - f[0]) * RT * 9 / 5
        else:
            u = (sum(x * b for x, b in zip(XU9, f)) + hdt * force[0]) / (rho * RT)
            v = (sum(x * b for x, b in zip(XV9, f)) + hdt * force[1]) / (rho * RT)
            p = sum(f) + hdt * RT * (grho[0] * u + grho[1] * v)
        # sources of the next step; the rows beyond a wall are those of the step's start
        e = torch.cat([wrap(was, True)[:1], phi, wrap(was, True)[-1:]]) if walls else wrap(phi, False)
        gx, gyy = (torch.where(k.abs() < 1e-14, zero, k) for k in iso_gradient(e))
        n, s = e[2:], e[:-2]
        lap = (4 * (east(phi) + west(phi) + n + s) + east(n) + west(n) + east(s) + west(s) - 20 * phi) / 6
        mu = 2 * beta * (phi - 1) * phi * (2 * phi - 1) - kappa * lap
        grho, force = [a_phi * gx, a_phi * gyy], [mu * gx, mu * gyy]
        if gy:
            force[1] = force[1] - gy * (rho - kw['RhoL'])
        norm = torch.sqrt(gx * gx + gyy * gyy)
        k = torch.where(norm > 0, -4 * (phi - 1) * phi / kw['W'] / torch.where(norm > 0, norm, 1.0), zero)
        now = (phi * u, phi * v)
        src = [gx * k + (now[0] - old[0]) / (RT * dt), gyy * k + (now[1] - old[1]) / (RT * dt)]
        old = now
    return dict(rho=rho, u=u, v=v, phi=phi, p=p)


def d2v16_matrix(c):
    """The inverse of the 16 moments' basis; the first ring carries an internal speed 3c."""
    xu, xv = c * np.array(XU16, float), c * np.array(XV16, float)
    x2 = xu ** 2 + xv ** 2 + np.array([9 * c * c] * 4 + [0.0] * 12)
    return np.linalg.inv(np.array([np.ones(16), xu, xv, x2, xu * xv, xu ** 2, xv ** 2, xu * x2, xv * x2, xu ** 3,
                                   xv ** 3, xu ** 2 * xv, xu * xv ** 2, xu * xv * x2, xu ** 2 * x2, xv ** 2 * x2]))


def pp_equilibrium(model, kw, rho, u, v):
    if model == 'PP9':
        out = []
        for q in range(9):
            u1 = (XU9[q] * u + XV9[q] * v) / RT
            out.append(W9[q] * rho * (1 + u1 + 0.5 * u1 * u1 - (u * u + v * v) / (2 * RT)))
        return out
    p, u2, v2 = rho * RT, u * u, v * v
    s2 = u2 + v2
    m = [rho, rho * u, rho * v, rho * (3 * RT + s2), rho * u * v, rho * u2 + p, rho * v2 + p,
         rho * u * (5 * RT + s2), rho * v * (5 * RT + s2), rho * u * (3 * RT + u2), rho * v * (3 * RT + v2),
         rho * v * (RT + u2), rho * u * (RT + v2), (7 * RT + s2) * rho * u * v,
         5 * rho * RT * RT + p * (8 * u2 + v2) + rho * u2 * s2, 5 * rho * RT * RT + p * (8 * v2 + u2) + rho * v2 * s2]
    a = torch.from_numpy(d2v16_matrix(kw['d2v16_c'])).to(rho.device)
    return list(torch.einsum('jk,kyx->jyx', a, torch.stack(m)))


def pp_run(model, kw, st, steps):
    """Pseudopotential models (periodic): `steps` steps from the state `st`."""
    if model == 'PP9':
        xu, xv, dt = XU9, XV9, 0.5
    else:
        c = kw['d2v16_c']
        xu, xv, dt = [c * k for k in XU16], [c * k for k in XV16], 0.5 / (2 * c * math.sqrt(2.0))
    hdt, tau = 0.5 * dt, kw['Mu0'] / RT
    t_cs, a_cs = kw['Tr'] * kw.get('Tc_CS', 0.0943), kw.get('aCS', 1.0)

    def pressure(r):
        return r * t_cs * (1 + r + r ** 2 - r ** 3) / (1 - r) ** 3 - a_cs * r * r

    def psi_of(r):
        d = pressure(r) - r * RT
        return torch.sqrt(2 * d.abs()), torch.sign(d)

    f, rho, u, v = st['f'], st['rho'], st['u'], st['v']
    zero = torch.zeros_like(rho)
    force, face_force = (zero, zero), [(zero, zero), (zero, zero)]
    a, b = (2 * tau - hdt) / (2 * tau + dt), 2 * tau / (2 * tau + hdt)

    def relax(coef, old, r, uu, vv, fx, fy):
        eq = pp_equilibrium(model, kw, r, uu, vv)
        return [coef * o + (1 - coef) * e * (1 + tau * (fx * (x - uu) + fy * (y - vv)) / (r * RT))
                for o, e, x, y in zip(old, eq, xu, xv)]

    for _ in range(steps):
        bf = relax(a, f, rho, u, v, *force)
        net = [zero] * len(f)
        for d, along_x in enumerate((True, False)):
            g = [face_value(bf[q], False, xu[q], xv[q], hdt, along_x, 'CD')[:len(rho)] for q in range(len(f))]
            r = sum(g)
            uu = (sum(x * k for x, k in zip(xu, g)) + 0.5 * hdt * face_force[d][0]) / r
            vv = (sum(x * k for x, k in zip(xv, g)) + 0.5 * hdt * face_force[d][1]) / r
            psi, sign = psi_of(r)
            face_force[d] = tuple(-sign * psi * k for k in iso_gradient(wrap(psi, False)))
            g = relax(b, g, r, uu, vv, *face_force[d])
            for q, k in enumerate(g):
                k = k * (xu[q] if along_x else xv[q])
                net[q] = net[q] + dt * (k - (east(k) if along_x else torch.roll(k, -1, 0)))
        f = [4 / 3 * bf[q] - f[q] / 3 + net[q] for q in range(len(f))]
        rho = sum(f)
        u = (sum(x * k for x, k in zip(xu, f)) + hdt * force[0]) / rho
        v = (sum(x * k for x, k in zip(xv, f)) + hdt * force[1]) / rho
        psi, sign = psi_of(rho)
        force = tuple(-sign * psi * k for k in iso_gradient(wrap(psi, False)))
    return dict(rho=rho, u=u, v=v, p=pressure(rho))


def exact(case, seed):
    if case['kind'] == 'serve':
        out = []
        for k, r in enumerate(serving_requests(case, seed)):
            if k >= 4:  # the rest would take minutes
                out.append([None, None])
                continue
            st = initial_state(r['model'], r['kw'], r['init'], r['params'], seed % (1 << 32) + 1 + k, r['n'], r['n'])
            if r['model'] == 'AC':
                got = ac_run('AC', r['kw'], False, 'CD', st, case['steps'])
                out.append([got['rho'], got['phi']])
            else:
                got = pp_run('PP16', r['kw'], st, case['steps'])
                out.append([got['rho'], got['u']])
        return out
    kw, walls, _, _ = physics(case, seed)
    st = initial(case, seed)
    if case['model'] in ('PP9', 'PP16'):
        got = pp_run(case['model'], kw, st, case['steps'])
    else:
        got = ac_run(case['model'], kw, walls, case.get('scheme', 'CD'), st, case['steps'])
        got['sum_phi'] = float(got['phi'].sum())
    got['sum_rho'] = float(got['rho'].sum())
    return got
