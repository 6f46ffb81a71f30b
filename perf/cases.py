"""The work a user of the solver has it do, as cases that can be timed.

A case is a dict of plain values. Its ``kind`` is the entry point it goes
through: the drop-in ``step`` of the host loop, the graph-replayed ``run``, a
``batch.Batch`` of a parameter scan, the stage functions ``deposit`` and
``calculate_*``, and the gradients of a training sample of the field
predictor. Inputs are smooth random plasma states in the solver's own units
(lengths in plasma skin depths): fields, densities, displacements and momenta
of relative size ``drive``, varying over about one unit, which is what the
solver meets between a weakly driven wake (0.01) and a blowout (0.3).
``exact`` restates the step, the stages and the network in plain float64
torch.

The transform forms that the framework keeps for comparison (split-bf16,
split-tf32) are slower and less accurate than the float64 FFT form, so nobody
picks them for a run: the forms here are the default (FFT where 2(N - 1)
factors into 2, 3, 5, dense transforms elsewhere) and float32 FFT transforms.
"""
import math
import types

import numpy as np
import torch

from lcode3d_b200 import batch as B
from lcode3d_b200 import lcode as L
from lcode3d_b200 import predictor as P

PARTS = ('x_offt', 'y_offt', 'px', 'py', 'pz')
FIELDS = ('Ex', 'Ey', 'Ez', 'Bx', 'By', 'Bz')
DENSITIES = ('ro', 'jx', 'jy', 'jz')
STATE = PARTS + FIELDS + DENSITIES
COARSENESS, FINENESS, PADDING = 3, 2, 10
RUN_BEAM = (0.5, 1.0, 1.0)


def listed():
    return [
        # the smallest grid in use (trial runs, tests): nothing but launches and host work
        dict(name='step_41', kind='step', N=41, h=0.1, drive=0.05, precision='fp64'),
        # a small production grid in the host loop (weakly driven wake)
        dict(name='step_161', kind='step', N=161, h=0.05, drive=0.05, precision='fp64'),
        # the production grid in the host loop, blowout regime
        dict(name='step_641', kind='step', N=641, h=0.025, drive=0.2, precision='fp64'),
        # a fine grid, the largest that users of one GPU are likely to run
        dict(name='step_1025', kind='step', N=1025, h=16 / 1024, drive=0.2, precision='fp64'),
        # a grid size chosen without regard to its factors (2 * 386 = 4 * 193): dense transforms
        dict(name='step_387', kind='step', N=387, h=16 / 386, drive=0.1, precision='fp64'),
        # the production grid with float32 transforms, the fastest form within 1e-6
        dict(name='step_641_fft32', kind='step', N=641, h=0.025, drive=0.2, precision='fft32'),
        # a middle-sized simulation run without host work between the steps
        dict(name='run_481', kind='run', N=481, h=16 / 480, drive=0.1, precision='fp64', steps=16),
        # a small one: what a quick look at a parameter set costs
        dict(name='run_161', kind='run', N=161, h=0.1, drive=0.05, precision='fp64', steps=32),
        # a parameter scan over the grid sizes that scans draw from
        dict(name='scan_8', kind='scan', grids='161,161,321,321,481,481,641,641', steps=8),
        # the deposition stage on its own, strongly disturbed plasma
        dict(name='deposit_641', kind='deposit', N=641, h=0.025, drive=0.3, precision='fp64'),
        # the three field solvers on their own, on a coarse grid
        dict(name='fields_321', kind='fields', N=321, h=0.05, drive=0.1, precision='fp64'),
        # the gradients of one training sample of the field predictor at the production size
        dict(name='train_641', kind='train', N=641),
    ]


def _smooth(n):
    for f in (2, 3, 5):
        while n % f == 0:
            n //= f
    return n == 1


SMOOTH = [n + 1 for n in range(40, 1025, 2) if _smooth(n)]   # grid sizes with FFT transforms


def _draw_size(rng, lo, hi, any_size):
    """An odd grid size, uniform over the logarithm: usually one with FFT
    transforms, as users are told to choose, else any."""
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    if any_size and rng.random() < 0.2:
        return min(2 * int(n / 2) + 1, 641)
    return min((s for s in SMOOTH if lo <= s <= hi), key=lambda s: abs(math.log(s / n)))


def draw(rng):
    kind = rng.choice(('step', 'step', 'step', 'step', 'run', 'run', 'scan', 'deposit', 'fields', 'train'))
    drive = round(math.exp(rng.uniform(math.log(0.01), math.log(0.3))), 4)
    if kind == 'scan':
        grids = [rng.choice(B.GRIDS) for _ in range(rng.randint(2, 8))]
        return dict(kind='scan', grids=','.join(map(str, sorted(grids))), steps=rng.randint(2, 6))
    if kind == 'train':
        return dict(kind='train', N=_draw_size(rng, 41, 641, True))
    N = _draw_size(rng, 41, 1025 if kind in ('step', 'deposit', 'fields') else 641, kind in ('step', 'deposit'))
    h = round(rng.uniform(8.0, 20.0) / (N - 1), 5) if N > 100 else 0.1
    case = dict(kind=kind, N=N, h=h, drive=drive, precision='fp64')
    if kind == 'step' and N in SMOOTH and rng.random() < 0.3:
        case['precision'] = 'fft32'
    if kind == 'run':
        case['steps'] = rng.randint(2, 8)
    return case


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------

_plasmas = {}   # one plasma layout (config, const, virt_params) per configuration, as a program keeps it


def _config(case):
    c = types.SimpleNamespace(
        grid_steps=case['N'], grid_step_size=case['h'], xi_step_size=round(0.2 * case['h'], 6), xi_steps=10 ** 9,
        diagnostics_each_N_steps=10 ** 9, field_solver_subtraction_trick=1, field_solver_variant_A=True,
        reflect_padding_steps=5, plasma_padding_steps=PADDING, plasma_coarseness=COARSENESS,
        plasma_fineness=FINENESS, gpu_index=0, lc3d_precision=case['precision'])
    c.reflect_boundary = c.grid_step_size * (c.grid_steps / 2 - c.reflect_padding_steps)
    return c


def _plasma(case):
    key = (case['N'], case['h'], case['precision'])
    if key not in _plasmas:
        if len(_plasmas) >= 4:
            _plasmas.clear()
        cfg = _config(case)
        xs, ys, const, virt, _ = L.init(cfg)
        _plasmas[key] = cfg, const, virt
    return _plasmas[key]


class _Waves:
    """Smooth random functions of (x, y): sums of plane waves of about one
    unit's length, of unit root mean square."""

    def __init__(self, seed):
        self.gen = torch.Generator().manual_seed(int(seed))

    def uniform(self, lo, hi, n=1):
        return lo + (hi - lo) * torch.rand(n, generator=self.gen, dtype=torch.float64)

    def __call__(self, x, y, amplitude):
        n = 12
        k, ang = self.uniform(0.4, 2.2, n), self.uniform(0, 2 * math.pi, n)
        phase = self.uniform(0, 2 * math.pi, n)
        out = torch.zeros_like(x)
        for a, b, p in zip((k * ang.cos()).tolist(), (k * ang.sin()).tolist(), phase.tolist()):
            out += torch.sin(a * x + b * y + p)
        return out * (amplitude / math.sqrt(n / 2))


def _coords(n, step):
    x = (torch.arange(n, dtype=torch.float64, device='cuda') - n // 2) * step
    return x[:, None].expand(n, n).contiguous(), x[None, :].expand(n, n).contiguous()


def _make_state(case, waves):
    """The 15 arrays of a state: plasma displaced and moving smoothly, at
    rest at the plasma's edge."""
    N, h, d = case['N'], case['h'], case['drive']
    X, Y = _coords(N, h)
    Nc = 2 * ((N - 2 * PADDING) // (2 * COARSENESS)) - 1
    x, y = _coords(Nc, COARSENESS * h)
    edge = max(float(x.max()), COARSENESS * h)
    taper = (1 - (x / edge) ** 8) * (1 - (y / edge) ** 8)
    m = COARSENESS ** 2
    move = 0.7 * d * min(1.0, edge / 8)
    s = {'x_offt': waves(x, y, move) * taper, 'y_offt': waves(x, y, move) * taper,
         'px': waves(x, y, m * d) * taper, 'py': waves(x, y, m * d) * taper,
         'pz': (waves(x, y, 0.4 * m * d) + 0.5 * m * d * d) * taper}
    for n in FIELDS + DENSITIES:
        s[n] = waves(X, Y, d)
    return s


def _beam(case, waves):
    """The driver's charge density of one step, in pinned host memory (the
    host loop evaluates it there)."""
    N, h = case['N'], case['h']
    x = (np.arange(N) - N // 2) * h
    xi = float(waves.uniform(1.0, 4.0))
    b = case['drive'] * np.exp(-(x[:, None] ** 2 + x[None, :] ** 2) / 2) * 0.5 * (1 - math.cos(math.sqrt(math.pi / 2) * xi))
    return torch.from_numpy(b).pin_memory()


def _specs(case, seed):
    rng = np.random.default_rng(seed)
    return [dict(grid_steps=int(N), grid_step_size=16.0 / (int(N) - 1), xi_step_size=0.01,
                 amplitude=float(np.exp(rng.uniform(np.log(0.05), np.log(1.0)))),
                 sigma_r=float(rng.uniform(0.5, 2.0)), length_factor=float(rng.uniform(0.5, 1.5)))
            for N in case['grids'].split(',')]


def _train_fields(case, waves):
    """The fields of the two previous steps and the first-pass fields of the
    next: a smooth state, a small change of it, a still smaller one."""
    X, Y = _coords(case['N'], 16.0 / (case['N'] - 1))
    f2 = {n: waves(X, Y, 0.1) for n in FIELDS + DENSITIES}
    f1 = {n: f2[n] + waves(X, Y, 1e-3) for n in FIELDS + DENSITIES}
    first = {n: 2 * f1[n] - f2[n] + waves(X, Y, 2e-4) for n in FIELDS}
    return types.SimpleNamespace(**f1), types.SimpleNamespace(**f2), first


def prepare(case, seed):
    s = types.SimpleNamespace(kind=case['kind'], case=case)
    waves = _Waves(seed)
    if case['kind'] == 'scan':
        s.batch = B.Batch(_specs(case, seed))
        return s
    if case['kind'] == 'train':
        s.f1, s.f2, s.first = _train_fields(case, waves)
        s.net = P.FieldPredictor(case['N'], seed=seed)
        s.net.pack(s.f1, s.f2)
        s.net.set_target(s.first, s.f1, s.f2)
        s.sample = P.Sample(s.net.buffer('input').clone(), s.net.buffer('target').clone())
        return s
    s.cfg, s.const, s.virt = _plasma(case)
    a = _make_state(case, waves)
    s.state = L.GPUArrays(**a)
    if case['kind'] == 'step':
        s.beam = _beam(case, waves)
    elif case['kind'] == 'fields':
        X, Y = _coords(case['N'], case['h'])
        s.beam = case['drive'] * torch.exp(-(X ** 2 + Y ** 2) / 2)
        s.j_prev = [getattr(s.state, n) * 0.99 for n in ('jx', 'jy')]
    return s


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------

def run(s):
    if s.kind == 'step':
        new = L.step(s.cfg, s.const, s.virt, s.state, s.beam)
        return {n: getattr(new, n) for n in STATE}
    if s.kind == 'run':
        new, ez = L.run(s.cfg, s.const, s.virt, s.state, 100, s.case['steps'], RUN_BEAM)
        return dict({n: getattr(new, n) for n in STATE}, history=ez)
    if s.kind == 'scan':
        return s.batch.run(s.case['steps'])
    if s.kind == 'train':
        net = s.net
        net.buffer('input').copy_(s.sample.x)
        net.buffer('target').copy_(s.sample.t)
        net.forward()
        net.backward()
        N = net.N   # the output is the network's own memory, freed with it: a copy goes out
        return {'grad': net.grad(), 'output': net.buffer('output').view(N, N + 1, 16)[:, :N, :P.N_OUT].clone()}
    st = s.state
    if s.kind == 'deposit':
        return L.deposit(s.cfg, s.const.ro_initial, *[getattr(st, n) for n in PARTS[:2]], s.const.m, s.const.q,
                         st.px, st.py, st.pz, s.virt)
    transverse = L.calculate_Ex_Ey_Bx_By(s.cfg, st.Ex, st.Ey, st.Bx, st.By, s.beam, st.ro, st.jx, st.jy, st.jz,
                                         *s.j_prev)
    return [*transverse, L.calculate_Ez(s.cfg, st.jx, st.jy), L.calculate_Bz(s.cfg, st.jx, st.jy)]


# ---------------------------------------------------------------------------
# Work a pass cannot do without
# ---------------------------------------------------------------------------

def _solve_flops(N):
    """Six fields, four 1-D real transforms along each of N rows."""
    return 6 * 4 * N * 2.5 * N * math.log2(N) + 60 * N * N


def _step_work(N):
    Nc = 2 * ((N - 2 * PADDING) // (2 * COARSENESS)) - 1
    fine = ((N - 2 * PADDING) // 2 * FINENESS * 2) ** 2
    return {'bytes': 8.0 * (2 * (5 * Nc * Nc + 10 * N * N) + 4 * Nc * Nc + 2 * N * N),
            'flops': 3 * (130.0 * fine + 230.0 * Nc * Nc) + 2 * _solve_flops(N)}


def work(case):
    kind = case['kind']
    if kind == 'scan':
        each = [_step_work(int(N)) for N in case['grids'].split(',')]
        return {'bytes': sum(w['bytes'] for w in each), 'flops': case['steps'] * sum(w['flops'] for w in each)}
    N = case['N']
    w = _step_work(N)
    if kind == 'run':
        return {'bytes': w['bytes'], 'flops': case['steps'] * w['flops']}
    if kind == 'deposit':
        Nc = 2 * ((N - 2 * PADDING) // (2 * COARSENESS)) - 1
        return {'bytes': 8.0 * (7 * Nc * Nc + 5 * N * N), 'flops': 130.0 * ((N - 2 * PADDING) // 2 * FINENESS * 2) ** 2}
    if kind == 'fields':
        return {'bytes': 8.0 * (13 + 4 + 6) * N * N, 'flops': _solve_flops(N)}
    if kind == 'train':
        pixels = [N * N, ((N + 1) // 2) ** 2, ((N + 3) // 4) ** 2]
        macs = sum(9 * ci * co * pixels[k] for (ci, co), k in zip(P.LAYERS, (0, 1, 2, 2, 1, 0)))
        return {'bytes': 2.0 * 32 * N * N + 2 * 4.0 * 16 * N * N + 16.0 * 198480, 'flops': 6.0 * macs}
    return w


# ---------------------------------------------------------------------------
# The same in plain float64 torch
# ---------------------------------------------------------------------------

def _dst(N):
    """2 sin(pi k n / (N - 1)), k, n = 1 .. N-2."""
    k = torch.arange(1, N - 1, device='cuda')
    r = (k[:, None] * k[None, :]) % (2 * (N - 1))
    return 2 * torch.sin(r.double() * (math.pi / (N - 1)))


def _dct(N):
    """c_n cos(pi k n / (N - 1)), c = 1 at the ends, else 2; k, n = 0 .. N-1."""
    k = torch.arange(N, device='cuda')
    r = (k[:, None] * k[None, :]) % (2 * (N - 1))
    w = torch.full((N,), 2.0, dtype=torch.float64, device='cuda')
    w[0] = w[-1] = 1
    return torch.cos(r.double() * (math.pi / (N - 1))) * w[None, :]


class _Exact:
    """The xi step and its stages at one grid size."""

    def __init__(self, N, h, dxi):
        self.N, self.h, self.dxi = N, h, dxi
        self.rb = h * (N / 2 - 5)
        S, C = _dst(N), _dct(N)
        k = torch.arange(N, dtype=torch.float64, device='cuda')
        lam = 4 / h ** 2 * torch.sin(k * math.pi / (2 * (N - 1))) ** 2
        norm = (2.0 * (N - 1)) ** 2
        li = lam[1:-1]
        mix = 1 / (li[:, None] + lam[None, :] + 1) / norm
        neu = lam[:, None] + lam[None, :]
        neu[0, 0] = math.inf
        self.solve_sd = lambda a: S @ (mix * (S @ a @ C.T)) @ C.T               # (N-2) x N
        self.solve_ds = lambda a: C @ (mix.T * (C @ a @ S)) @ S                 # N x (N-2)
        self.solve_ss = lambda a: S @ ((S @ a @ S) / (li[:, None] + li[None, :]) / norm) @ S
        self.solve_cc = lambda a: C @ ((C @ a @ C.T) / neu / norm) @ C.T
        # plasma lattices
        steps = N - 2 * PADDING
        half = torch.arange(steps // (2 * COARSENESS), dtype=torch.float64, device='cuda') * (h * COARSENESS)
        self.coarse = coarse = torch.cat([-half[1:].flip(0), half])
        half = (.5 + torch.arange(steps // 2 * FINENESS, dtype=torch.float64, device='cuda')) * (h / FINENESS)
        self.fine = fine = torch.cat([-half.flip(0), half])
        n = len(coarse)
        pos = torch.searchsorted(coarse, fine)
        self.nxt, self.prv = pos.clamp(0, n - 1), (pos - 1).clamp(0, n - 1)
        self.wp, self.wn = (coarse[self.nxt] - fine) / (h * COARSENESS), (fine - coarse[self.prv]) / (h * COARSENESS)
        low, high = self.nxt == 0, self.prv == n - 1
        self.wp[low], self.wn[low], self.wn[high], self.wp[high] = 0, 1, 0, 1
        z = torch.zeros((n, n), dtype=torch.float64, device='cuda')
        self.x0, self.y0 = z + coarse[:, None], z + coarse[None, :]
        self.m, self.q = z + COARSENESS ** 2, z - COARSENESS ** 2
        self.ions = 0
        self.ions = -self.deposit(z, z, z, z, z)[0]

    def _cells(self, x, y):
        xh, yh = x / self.h + .5, y / self.h + .5
        i, j = xh.floor(), yh.floor()
        a, b = xh - i - .5, yh - j - .5
        wx = ((.5 - a) ** 2 / 2, .75 - a ** 2, (.5 + a) ** 2 / 2)
        wy = ((.5 - b) ** 2 / 2, .75 - b ** 2, (.5 + b) ** 2 / 2)
        return (i.long() + self.N // 2) * self.N + j.long() + self.N // 2, wx, wy

    def deposit(self, x_offt, y_offt, px, py, pz):
        wp, wn = self.wp, self.wn

        def mix(c):
            rows = wp[:, None] * c[self.prv] + wn[:, None] * c[self.nxt]
            return wp[None, :] * rows[:, self.prv] + wn[None, :] * rows[:, self.nxt]
        x, y = self.fine[:, None] + mix(x_offt), self.fine[None, :] + mix(y_offt)
        m, q, px, py, pz = (mix(v) / (COARSENESS * FINENESS) ** 2 for v in (self.m, self.q, px, py, pz))
        gamma_m = torch.sqrt(m ** 2 + px ** 2 + py ** 2 + pz ** 2)
        ro = q / (1 - pz / gamma_m)
        vals = (ro, px * (ro / gamma_m), py * (ro / gamma_m), pz * (ro / gamma_m))
        cell, wx, wy = self._cells(x, y)
        out = [torch.zeros(self.N * self.N, dtype=torch.float64, device='cuda') for _ in vals]
        for di in range(3):
            for dj in range(3):
                at = (cell + (di - 1) * self.N + dj - 1).reshape(-1)
                w = wx[di] * wy[dj]
                for o, v in zip(out, vals):
                    o.index_add_(0, at, (v * w).reshape(-1))
        out = [o.view(self.N, self.N) for o in out]
        return [out[0] + self.ions, *out[1:]]

    def _reflect(self, x):
        x = torch.where(x > self.rb, 2 * self.rb - x, x)
        return torch.where(x < -self.rb, -2 * self.rb - x, x)

    def estimate(self, s):
        g = torch.sqrt(self.m ** 2 + s['pz'] ** 2 + s['px'] ** 2 + s['py'] ** 2)
        x = self.x0 + s['x_offt'] + s['px'] / (g - s['pz']) * self.dxi
        y = self.y0 + s['y_offt'] + s['py'] / (g - s['pz']) * self.dxi
        return self._reflect(x) - self.x0, self._reflect(y) - self.y0

    def move(self, s, est, fields):
        cell, wx, wy = self._cells(self.x0 + (s['x_offt'] + est[0]) / 2, self.y0 + (s['y_offt'] + est[1]) / 2)

        def gather(a):
            a = a.reshape(-1)
            return sum(a[cell + (di - 1) * self.N + dj - 1] * (wx[di] * wy[dj]) for di in range(3) for dj in range(3))
        Ex, Ey, Ez, Bx, By, Bz = (gather(fields[n]) for n in FIELDS)
        px, py, pz = s['px'], s['py'], s['pz']
        for _ in range(2):
            g = torch.sqrt(self.m ** 2 + pz ** 2 + px ** 2 + py ** 2)
            vx, vy, vz = px / g, py / g, pz / g
            k = self.q * self.dxi / (1 - pz / g)
            dpx, dpy, dpz = (k * (Ex + vy * Bz - vz * By), k * (Ey - vx * Bz + vz * Bx), k * (Ez + vx * By - vy * Bx))
            px, py, pz = s['px'] + dpx / 2, s['py'] + dpy / 2, s['pz'] + dpz / 2
        g = torch.sqrt(self.m ** 2 + pz ** 2 + px ** 2 + py ** 2)
        x = self.x0 + s['x_offt'] + px / (g - pz) * self.dxi
        y = self.y0 + s['y_offt'] + py / (g - pz) * self.dxi
        px, py, pz = s['px'] + dpx, s['py'] + dpy, s['pz'] + dpz
        px, py = (torch.where(v.abs() > self.rb, -p, p) for v, p in ((x, px), (y, py)))
        return {'x_offt': self._reflect(x) - self.x0, 'y_offt': self._reflect(y) - self.y0, 'px': px, 'py': py, 'pz': pz}

    def _dx(self, a):
        return (a[2:, 1:-1] - a[:-2, 1:-1]) / (2 * self.h)

    def _dy(self, a):
        return (a[1:-1, 2:] - a[1:-1, :-2]) / (2 * self.h)

    def transverse(self, sub, beam, ro, jx, jy, jz, jx_prev, jy_prev):
        def grow(a):
            return torch.nn.functional.pad(a, (1, 1, 1, 1))
        jx_xi, jy_xi = (jx_prev - jx) / self.dxi, (jy_prev - jy) / self.dxi
        ro, jz = ro + beam, jz + beam
        rhs = {'Ex': -((grow(self._dx(ro)) - jx_xi) - sub['Ex']), 'Ey': -((grow(self._dy(ro)) - jy_xi) - sub['Ey']),
               'Bx': (grow(self._dy(jz)) - jy_xi) + sub['Bx'], 'By': -((grow(self._dx(jz)) - jx_xi) - sub['By'])}
        out = {}
        for n in ('Ex', 'By'):
            out[n] = torch.nn.functional.pad(self.solve_ds(rhs[n][:, 1:-1]), (1, 1))
        for n in ('Ey', 'Bx'):
            out[n] = torch.nn.functional.pad(self.solve_sd(rhs[n][1:-1]), (0, 0, 1, 1))
        return out

    def longitudinal(self, jx, jy):
        Ez = torch.nn.functional.pad(self.solve_ss(-(self._dx(jx) + self._dy(jy))), (1, 1, 1, 1))
        Bz = self.solve_cc(torch.nn.functional.pad(-(self._dy(jx) - self._dx(jy)), (1, 1, 1, 1)))
        return {'Ez': Ez, 'Bz': Bz - Bz.mean()}

    def step(self, s, beam):
        est, avg, sub = self.estimate(s), s, s
        for _ in range(2):
            p = self.move(s, est, avg)
            est = p['x_offt'], p['y_offt']
            ro, jx, jy, jz = self.deposit(**p)
            F = self.transverse(sub, beam, (ro + s['ro']) / 2, jx, jy, (jz + s['jz']) / 2, s['jx'], s['jy'])
            F = {n: 2 * F[n] - s[n] for n in F}
            F.update(self.longitudinal(jx, jy))
            avg = sub = {n: (F[n] + s[n]) / 2 for n in FIELDS}
        p = self.move(s, est, avg)
        return {**p, **F, **dict(zip(DENSITIES, self.deposit(**p)))}

    def beam(self, xi_i, amplitude, sigma, length):
        xi = xi_i * self.dxi
        x, y = _coords(self.N, self.h)
        if not 0 <= xi <= 2 * math.sqrt(2 * math.pi) * length:
            return torch.zeros_like(x)
        return amplitude * torch.exp(-(x ** 2 + y ** 2) / (2 * sigma ** 2)) * 0.5 * (
            1 - math.cos(math.sqrt(math.pi / 2) * xi / length))

    def run(self, s, xi0, steps, beam):
        ez = []
        for k in range(steps):
            s = self.step(s, self.beam(xi0 + k, *beam))
            ez.append(s['Ez'][self.N // 2, self.N // 2])
        return s, torch.stack(ez)


def _exact_train(case, seed, waves):
    """Forward pass and gradients of the network in float64 (the training
    kernels keep its activations in bfloat16)."""
    N, F = case['N'], torch.nn.functional
    f1, f2, first = _train_fields(case, waves)
    a = [getattr(f1, n) for n in P.FIELDS_IN]
    d = [u - getattr(f2, n) for u, n in zip(a, P.FIELDS_IN)]
    scales = [v.square().mean().sqrt() for v in a + d]
    out_scale = torch.stack(scales[13:18]).square().mean().sqrt()
    x = torch.zeros((1, 32, N, N), dtype=torch.float64, device='cuda')
    for c in range(18):
        x[0, c] = (a + d)[c] / scales[c]
    for c in range(9):
        x[0, 18 + c] = scales[c].log10() / 4
    t = torch.stack([first[n] - (2 * getattr(f1, n) - getattr(f2, n)) for n in P.FIELDS_OUT]) / out_scale
    flat = torch.from_numpy(P.init_params(seed)).cuda().double().requires_grad_()
    layers, at = [], 0
    for ci, co in P.LAYERS:
        w = flat[at:at + 9 * co * ci].view(3, 3, co, ci).permute(2, 3, 0, 1)
        layers.append((w, flat[at + 9 * co * ci:at + 9 * co * ci + co]))
        at += 9 * co * ci + co

    def conv(v, k):
        """The convolution as nine products of shifted images (plain float64)."""
        w, b = layers[k]
        p = F.pad(v, (1, 1, 1, 1))
        H, W = v.shape[2:]
        y = sum(torch.einsum('oi,ihw->ohw', w[:, :, i, j], p[0, :, i:i + H, j:j + W]) for i in range(3) for j in range(3))
        return (y + b[:, None, None])[None]

    def pool(v):
        return F.avg_pool2d(v, 2, ceil_mode=True)

    def up(v, like):
        return v.repeat_interleave(2, 2).repeat_interleave(2, 3)[:, :, :like.shape[2], :like.shape[3]]
    e1 = conv(x, 0).relu()
    e2 = conv(pool(e1), 1).relu()
    e3 = conv(pool(e2), 2).relu()
    d2 = (up(conv(e3, 3), e2) + e2).relu()
    d1 = (up(conv(d2, 4), e1) + e1).relu()
    y = conv(d1, 5)[0, :P.N_OUT]
    (y - t).square().mean().backward()
    return {'grad': flat.grad, 'output': y.detach().permute(1, 2, 0).contiguous()}


def exact(case, seed):
    kind, waves = case['kind'], _Waves(seed)
    if kind == 'train':
        return _exact_train(case, seed, waves)
    if kind == 'scan':
        out = []
        for p in _specs(case, seed):
            e = _Exact(p['grid_steps'], p['grid_step_size'], p['xi_step_size'])
            n, zero = len(e.coarse), torch.zeros((e.N, e.N), dtype=torch.float64, device='cuda')
            s = dict({k: torch.zeros((n, n), dtype=torch.float64, device='cuda') for k in PARTS},
                     **{k: zero for k in FIELDS + DENSITIES})
            out.append(e.run(s, 0, case['steps'], (p['amplitude'], p['sigma_r'], p['length_factor']))[1])
        return out
    e = _Exact(case['N'], case['h'], _config(case).xi_step_size)
    s = _make_state(case, waves)
    if kind == 'step':
        return e.step(s, _beam(case, waves).cuda())
    if kind == 'run':
        new, ez = e.run(s, 100, case['steps'], RUN_BEAM)
        return dict(new, history=ez)
    if kind == 'deposit':
        return e.deposit(*[s[n] for n in PARTS])
    X, Y = _coords(case['N'], case['h'])
    F = e.transverse(s, case['drive'] * torch.exp(-(X ** 2 + Y ** 2) / 2), *[s[n] for n in DENSITIES],
                     0.99 * s['jx'], 0.99 * s['jy'])
    F.update(e.longitudinal(s['jx'], s['jy']))
    return [F[n] for n in ('Ex', 'Ey', 'Bx', 'By', 'Ez', 'Bz')]
