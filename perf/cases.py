"""Timed cases of the cavity solver: what its users have it do, through the public binding, on one GPU.

A pass advances cavities by a few time steps the way the callers do and leaves the complete state in a device
buffer the caller owns (`Cavity.checkpoint`, the snapshot a served or restarted run keeps):

* `interactive`: the run script's loop, one blocking step at a time, reading the probes after each and adding the
  mid-span statistics weighted with its dt (`Cavity.step`, `probes`, `add_statistics`);
* `queued`: the same outputs without a round trip per step (`step_outputs_async`, `sync_outputs`);
* `slots`: a server's round, a slot batch of cavities of one size with some slots free (`Batch`);
* `ensemble`: cavities of different sizes, Re and stretching stepped by one batch (`Batch`).

The state moves on from pass to pass, as a run does.  In the mixed form, whose fields are FP32, the potential is
handed on in FP32 too.  `exact` integrates the same equations in 64 bits with plain torch.
"""
import math

import numpy as np
import torch

from les_impulse3d_64_b200.api import Batch, Cavity

FIELDS = ('u', 'v', 'w', 'mx', 'my', 'mz')
LIDS = {'uniform': 0, 'regularised': 1, 'polynomial': 2}
PROBES = ((0.5, 0.5), (0.8, 0.8), (0.2, 0.2), (0.9, 0.1), (0.5, 0.9), (0.5, 0.1), (0.1, 0.5), (0.9, 0.5))
ENSEMBLE_SIZES = (24, 32, 48, 64)


def case(name, kind, n, nz, precision, steps, re, beta=0.0, lid='regularised', order=4, lag=False, fixed_dt=0.0,
         dx_wall=0.0, max_aspect=0.0, stats=False, count=1, slots=0):
    return dict(name=name, kind=kind, n=n, nz=nz, precision=precision, steps=steps, re=re, beta=beta, lid=lid,
                order=order, lag=lag, fixed_dt=fixed_dt, dx_wall=dx_wall, max_aspect=max_aspect, stats=stats,
                count=count, slots=slots)


def listed():
    return [
        # the reference's validation mesh, stepped interactively: the smallest run anyone makes
        case('validate_32x32x8_fp64', 'interactive', 32, 8, 'fp64', 8, 400.0, dx_wall=0.004, max_aspect=8.0),
        # the plain FP64 form on a uniform 32^3 grid, fixed dt
        case('plain_32cube_fp64', 'interactive', 32, 32, 'fp64', 8, 400.0, lid='polynomial', fixed_dt=2e-3),
        # the default benchmark size with probes and statistics every step, as the run script drives it
        case('plain_64cube_fp64', 'interactive', 64, 64, 'fp64', 8, 1000.0, beta=1.5, stats=True),
        # an odd box in the 2nd-order scheme with the lagged dt, outputs queued
        case('odd_50x50x37_fp64', 'queued', 50, 37, 'fp64', 8, 700.0, beta=1.3, order=2, lag=True, stats=True),
        # a finer FP64 run, axes beyond 64 cells and not multiples of a tile
        case('fine_100x100x75_fp64', 'queued', 100, 75, 'fp64', 8, 2000.0, beta=1.5),
        # the larger grids of the serving mix, each served alone
        case('serve_64x64x128_mixed', 'queued', 64, 128, 'mixed', 8, 1500.0, lid='uniform'),
        case('serve_96cube_mixed', 'queued', 96, 96, 'mixed', 8, 3000.0),
        # the mixed form at its benchmark size, and an odd box of that order
        case('mixed_128cube', 'queued', 128, 128, 'mixed', 8, 3200.0, beta=2.0),
        case('mixed_164x164x93', 'queued', 164, 93, 'mixed', 6, 2500.0, beta=1.2, lid='uniform'),
        # the largest benchmark size
        case('mixed_256cube', 'queued', 256, 256, 'mixed', 2, 3200.0, beta=2.0),
        # a server's round: one slot batch of 64^3 requests, one slot free
        case('slots_64cube_mixed', 'slots', 64, 64, 'mixed', 8, 1000.0, count=7, slots=8),
        # an uneven ensemble in one batch
        case('ensemble_24_to_64_mixed', 'ensemble', 0, 0, 'mixed', 8, 0.0, count=24),
    ]


def draw(rng):
    log = lambda lo, hi: math.exp(rng.uniform(math.log(lo), math.log(hi)))
    even = lambda v: 2 * max(3, round(v / 2))
    kind = rng.choice(('interactive', 'queued', 'queued', 'queued', 'slots', 'ensemble'))
    c = case('', kind, 0, 0, 'fp64', 8, round(log(200.0, 5000.0), 1),
             beta=rng.choice((0.0, round(rng.uniform(0.8, 2.0), 2))),
             lid=rng.choice(('uniform', 'regularised', 'regularised', 'polynomial')))
    del c['name']
    if kind == 'interactive':
        c.update(n=even(log(16, 72)), precision=rng.choice(('fp64', 'fp64', 'mixed')), stats=rng.random() < 0.5,
                 order=rng.choice((4, 4, 4, 2)), lag=rng.random() < 0.25)
        c['nz'] = max(6, round(c['n'] * rng.uniform(0.25, 1.4)))
    elif kind == 'queued':
        c.update(n=even(log(24, 200)), stats=rng.random() < 0.3, order=rng.choice((4, 4, 4, 4, 2)),
                 lag=rng.random() < 0.2)
        c['precision'] = rng.choice(('fp64', 'mixed')) if c['n'] <= 112 else 'mixed'
        c['nz'] = max(6, round(c['n'] * rng.uniform(0.4, 1.3)))
    elif kind == 'slots':
        c.update(n=even(log(24, 100)), precision='mixed', slots=8, count=rng.randint(3, 8))
        c['nz'] = max(6, round(c['n'] * rng.uniform(0.6, 1.5)))
    else:
        c.update(precision=rng.choice(('mixed', 'mixed', 'mixed', 'fp64')), count=rng.randint(6, 26), re=0.0, beta=0.0,
                 lid='regularised')
    cells = sum(s['nx'] * s['ny'] * s['nz'] for s in members(c))       # no more work than the largest listed case
    c['steps'] = max(1, min(8, int((2.4e7 if c['precision'] == 'mixed' else 1.4e7) / cells)))
    return c


# ------------------------------------------------------------------------------------------------ the members
def beta_wall_cell(n, beta):
    """First cell of an n-cell two-sided tanh grid on [0, 1] with clustering parameter beta."""
    return 0.5 * (1 + math.tanh(beta * (2.0 / n - 1)) / math.tanh(beta))


def settings_of(c, n, nz, re, beta):
    s = dict(nx=n, ny=n, nz=nz, lid_shaped=LIDS[c['lid']], impulse_order=c['order'], dt_lag=int(c['lag']),
             adaptive_dt=int(not c['fixed_dt']), phi_extrapolate=1, fdm_max_passes=8, fdm_rtol=1e-9, length=1.0, lz=1.0,
             u_lid=1.0, nu=1.0 / re, lid_ramp_t=0.0, reinit_r=0.98, impulse_order4_ramp=1.0,
             dt_fixed=c['fixed_dt'] or 2e-3, dt_max=4e-3, cfl_target=0.5, diffusion_limit=2.0, probes=PROBES,
             grid_stretch=0, grid_dx_wall=0.001, grid_max_aspect=c['max_aspect'])
    if beta or c['dx_wall']:
        s.update(grid_stretch=1, grid_dx_wall=c['dx_wall'] or beta_wall_cell(n, beta))
    return s


def members(c):
    """Settings of every cavity of a case."""
    if c['kind'] != 'ensemble':
        out = []
        for k in range(c['count']):      # requests of one size differ in Re and lid
            lid = dict(c, lid='uniform') if k % 2 else c
            out.append(settings_of(lid, c['n'], c['nz'], c['re'] * (1.0 + 0.5 * k), c['beta']))
        return out
    rng = np.random.default_rng(c['count'])
    out = []
    for k in range(c['count']):
        n = int(rng.choice(ENSEMBLE_SIZES))
        re = float(np.exp(rng.uniform(math.log(100.0), math.log(2000.0))))
        out.append(settings_of(c, n, n, re, 1.5 if k % 2 else 0.0))
    return out


def initial_noise(s, seed):
    """Gaussian noise of amplitude 1e-3 on v and w."""
    rng = np.random.default_rng(seed)
    nx, ny, nz = s['nx'], s['ny'], s['nz']
    return (1e-3 * rng.standard_normal((nz, ny + 1, nx)), 1e-3 * rng.standard_normal((nz + 1, ny, nx)))


def shapes_of(s):
    nx, ny, nz = s['nx'], s['ny'], s['nz']
    face = ((nz, ny, nx + 1), (nz, ny + 1, nx), (nz + 1, ny, nx))
    return face + face, (nz, ny, nx)


# ------------------------------------------------------------------------------------------------ one pass
class Snapshot:
    """A cavity's checkpoint in a device buffer, and typed views of its parts.  The parts of a checkpoint are
    256-byte aligned and end with u, v, w, mx, my, mz, phi, four potential increments and the statistics sums."""

    def __init__(self, cavity, s, precision):
        total = cavity.checkpoint_bytes()
        self.buffer = torch.zeros(total, dtype=torch.uint8, device='cuda')
        self.cavity, self.mixed = cavity, precision == 'mixed'
        dtype = torch.float32 if self.mixed else torch.float64
        width = 4 if self.mixed else 8
        face, cell = shapes_of(s)
        up = lambda b: (b + 255) // 256 * 256
        sizes = [up(width * math.prod(f)) for f in face] + [up(8 * math.prod(cell))] * 5 + [up(48 * cell[1] * cell[2])]
        at = total - sum(sizes)
        self.fields_at, self.parts = at, {}
        for name, f, size in zip(FIELDS, face, sizes):
            self.parts[name] = self.buffer[at:at + width * math.prod(f)].view(dtype).view(f)
            at += size
        self.fields = self.buffer[self.fields_at:at].view(dtype)
        self.parts['phi'] = self.buffer[at:at + 8 * math.prod(cell)].view(torch.float64).view(cell)
        self.sums = self.buffer[total - sizes[-1]:total - sizes[-1] + 48 * cell[1] * cell[2]].view(torch.float64)

    def take(self):
        self.cavity.checkpoint(self.buffer.data_ptr())

    def phi(self):
        return self.parts['phi'].float() if self.mixed else self.parts['phi']


class State:
    def __init__(self, c, seed):
        self.case, self.batch, self.cavities = c, None, []
        self.settings = members(c)
        for k, s in enumerate(self.settings):
            cavity = Cavity(s, precision=c['precision'])
            self.cavities.append(cavity)
            cavity.initialize(*initial_noise(s, seed * 64 + k))
        self.snapshots = [Snapshot(cav, s, c['precision']) for cav, s in zip(self.cavities, self.settings)]
        if c['kind'] in ('slots', 'ensemble'):
            self.batch = Batch(self.cavities, capacity=c['slots'] or None)

    def __del__(self):
        if self.batch is not None:
            self.batch.close()
        for cavity in self.cavities:
            cavity.close()


def prepare(c, seed):
    return State(c, seed)


def run(state):
    c = state.case
    if state.batch is not None:
        state.batch.step_async(c['steps'])
        reports = [r for r in state.batch.sync() if r is not None]
        out = dict(dt=np.array([r['dt'] for r in reports]), time=np.array([r['time'] for r in reports]),
                   steps=np.array([r['steps'] for r in reports]))
        for snap in state.snapshots:
            snap.take()
        out['fields'] = [snap.fields for snap in state.snapshots]
        out['phi'] = [snap.phi() for snap in state.snapshots]
        return out
    cavity, snap = state.cavities[0], state.snapshots[0]
    out = {}
    if c['kind'] == 'interactive':
        dt, probes, lines = [], [], []
        for _ in range(c['steps']):
            report = cavity.step()
            dt.append(report['dt'])
            probes.append(cavity.probes())
            if c['stats']:
                lines.append(cavity.add_statistics(report['dt']))
        out['dt'], out['probes'] = np.array(dt), np.array(probes)
        if c['stats']:
            out['lines'] = np.array(lines)
    else:
        cavity.step_outputs_async(c['steps'], c['stats'])
        report, out['probes'] = cavity.sync_outputs(c['steps'])
    snap.take()
    out.update({name: snap.parts[name] for name in FIELDS}, phi=snap.phi(), time=report['time'], steps=report['steps'])
    if c['stats']:
        out['sums'] = snap.sums
    return out


def work(c):
    """Algorithmic bytes and operations of a pass.  A stage of a step moves 18 face values (the sweep reads u, m and
    the RK base and writes the new impulse; the projection reads it for the divergence and the gradient and writes
    u), 72 bytes of potentials and 40 per pressure pass, per cell; the transforms take 4 (nx + ny + nz) operations
    per cell and pass and the stencils about 700.  From 128^3 cells the mixed form's FP32 transforms need a second
    pass to reach the tolerance."""
    total = {'bytes': 0.0, 'flops': 0.0}
    width = 4 if c['precision'] == 'mixed' else 8
    for s in members(c):
        cells = s['nx'] * s['ny'] * s['nz']
        passes = 2 if width == 4 and s['nx'] % 4 == 0 and cells >= 1 << 21 else 1
        total['bytes'] += c['steps'] * cells * (3.0 * (18 * width + 72 + 40 * passes) + 16)
        total['flops'] += c['steps'] * cells * 3.0 * (700 + 4 * passes * (s['nx'] + s['ny'] + s['nz']))
    return total


# ------------------------------------------------------------------------------------------------ in 64 bits
def axis_faces(n, dx_wall):
    if dx_wall >= 1.0 / n * (1 - 1e-12):
        f = np.arange(n + 1) * (1.0 / n)
        f[n] = 1.0
        return f
    xi = np.arange(n + 1) * (1.0 / n)
    xi[n] = 1.0
    lo, hi = 1e-8, 30.0
    for _ in range(200):
        b = 0.5 * (lo + hi)
        first = 0.5 * (1 + math.tanh(b * (2 * xi[1] - 1)) / math.tanh(b)) - 0.5 * (1 + math.tanh(-b) / math.tanh(b))
        lo, hi = (lo, b) if first < dx_wall else (b, hi)
    b = 0.5 * (lo + hi)
    f = 0.5 * (1 + np.tanh(b * (2 * xi - 1)) / math.tanh(b))
    f[0], f[n], f[n // 2] = 0.0, 1.0, 0.5
    return f


class Axis:
    """Grid of one axis (rounded to float, as the solver's tables are), the stencil tables of the Lamb vector at its
    faces, and the eigenbasis of its Neumann operator."""

    def __init__(self, s, n, device):
        ratio = lambda f: np.diff(f).max() / np.diff(f).min()
        if not s['grid_stretch']:
            f = axis_faces(n, 1e300)
        else:
            d = min(s['grid_dx_wall'], 1.0 / n)
            cap = s['grid_max_aspect']
            if cap > 0 and ratio(axis_faces(n, d)) > cap:
                lo, hi = d, 1.0 / n
                for _ in range(60):
                    mid = 0.5 * (lo + hi)
                    lo, hi = (mid, hi) if ratio(axis_faces(n, mid)) > cap else (lo, mid)
                d = hi
            f = axis_faces(n, d)
        w, c = np.diff(f), 0.5 * (f[1:] + f[:-1])
        sp = np.concatenate([[0.5 * w[0]], np.diff(c), [0.5 * w[-1]]])
        f, w, c, sp = (v.astype(np.float32).astype(np.float64) for v in (f, w, c, sp))
        self.n, self.face, self.w, self.c, self.sp = n, f, w, c, sp
        i = np.arange(n + 1)
        ramp = np.clip((np.minimum(i, n - i) - 1) / max(s['impulse_order4_ramp'], 1.0), 0.0, 1.0)
        narrow, wide = (i >= 1) & (i <= n - 1), (i >= 2) & (i <= n - 2)
        at = lambda v, k, ok: np.where(ok, v[np.clip(i + k, 0, n - 1)], 0.0)
        t = dict(inv_sp=1 / sp, ok=narrow.astype(float), l1=narrow * ramp, l3=wide * ramp)
        t['lo1'], t['hi1'] = at(w, -1, narrow) / (2 * sp), at(w, 0, narrow) / (2 * sp)
        both = np.where(wide, at(w, -2, wide) + at(w, 1, wide), 1.0)
        t['lo3'], t['hi3'] = at(w, -2, wide) / both, at(w, 1, wide) / both
        t['c3'] = np.where(wide, 0.5 * both / (2 * sp), 0.5)
        t['inv3'] = np.where(wide, 1 / np.where(wide, at(c, 1, wide) - at(c, -2, wide), 1.0), 0.0)
        root = np.sqrt(w)
        k = np.zeros((n, n))
        for j in range(n - 1):
            g = 1 / sp[j + 1]
            k[j, j] -= g
            k[j + 1, j + 1] -= g
            k[j, j + 1] = k[j + 1, j] = g
        lam, z = np.linalg.eigh(k / root[:, None] / root[None, :])
        lam[-1] = 0.0                          # the constant mode: the largest eigenvalue
        put = lambda v: torch.as_tensor(v, dtype=torch.float64, device=device)
        self.t = {key: put(v) for key, v in t.items()}
        self.width, self.lam, self.basis = put(w), put(lam), put(z / root[:, None])


class Exact:
    """One cavity's run in 64 bits: arrays are [z, y, x], axis a of the grid is dimension 2 - a."""

    def __init__(self, s, noise, device):
        self.s = s
        self.ax = [Axis(s, s[k], device) for k in ('nx', 'ny', 'nz')]
        self.device = device
        w = [a.width for a in self.ax]
        self.area = [self.along(w[(a + 1) % 3], (a + 1) % 3) * self.along(w[(a + 2) % 3], (a + 2) % 3) for a in range(3)]
        lam = self.along(self.ax[2].lam, 2) + self.along(self.ax[1].lam, 1) + self.along(self.ax[0].lam, 0)
        self.inv_lam = torch.where(lam == 0, torch.zeros_like(lam), 1 / torch.where(lam == 0, torch.ones_like(lam), lam))
        near = [min_pair(a.sp) for a in self.ax]
        geo = [np.float32(4.0) / (a.w.astype(np.float32) * m.astype(np.float32)) for a, m in zip(self.ax, near)]
        self.viscous = float(np.float32(s['nu']) * (geo[0].max() + geo[1].max() + geo[2].max()))
        fx, fz = self.ax[0].face, self.ax[2].c
        edge = lambda v: (1 - v ** 18) ** 2
        poly = lambda v: (v * (1 - v)) ** 2
        lid = {0: lambda: np.ones((len(fz), len(fx))), 1: lambda: edge(2 * fz - 1)[:, None] * edge(2 * fx - 1)[None],
               2: lambda: 16 * poly(fz)[:, None] * poly(fx)[None]}[s['lid_shaped']]()
        self.lid = torch.as_tensor(lid, device=device)
        self.time, self.dt, self.prev, self.count = 0.0, 0.0, None, 0
        put = lambda v: torch.as_tensor(v.astype(np.float32).astype(np.float64), device=device)
        nz, ny, nx = shapes_of(s)[1]
        self.m = [torch.zeros(nz, ny, nx + 1, dtype=torch.float64, device=device), put(noise[0]), put(noise[1])]
        for a in range(3):
            self.no_flow(self.m[a], a)
        self.u, self.phi = self.project(self.m)
        self.rate = self.cfl(self.u)
        self.sums = torch.zeros(6, ny, nx, dtype=torch.float64, device=device)

    @staticmethod
    def along(v, a):
        return v.view([-1 if d == 2 - a else 1 for d in range(3)])

    @staticmethod
    def no_flow(f, a):
        f.select(2 - a, 0).zero_()
        f.select(2 - a, f.shape[2 - a] - 1).zero_()

    def cut(self, f, a, lo, hi):
        """f at indices lo .. hi - 1 along axis a, repeated past its ends."""
        n = f.shape[2 - a]
        if 0 <= lo and hi <= n:
            return f.narrow(2 - a, lo, hi - lo)
        return f.index_select(2 - a, torch.arange(lo, hi, device=f.device).clamp(0, n - 1))

    def solve(self, r):
        s = [a.basis for a in self.ax]
        t = torch.matmul(s[1].T, torch.matmul(r, s[0]))
        t = torch.tensordot(s[2].T, t, dims=1) * self.inv_lam
        return torch.matmul(torch.matmul(s[1], torch.tensordot(s[2], t, dims=1)), s[0].T)

    def project(self, m):
        rhs = sum(torch.diff(m[a], dim=2 - a) * self.area[a] for a in range(3))
        phi = self.solve(rhs)
        left = rhs.clone()                      # once more on what rounding left
        for a in range(3):
            n = self.ax[a].n
            flux = torch.diff(phi, dim=2 - a) * self.along(self.ax[a].t['inv_sp'][1:n], a) * self.area[a]
            left.narrow(2 - a, 0, n - 1).sub_(flux)
            left.narrow(2 - a, 1, n - 1).add_(flux)
        phi = phi + self.solve(left)
        phi = phi - phi.mean()
        u = []
        for a in range(3):
            n = self.ax[a].n
            v = m[a].clone()
            v.narrow(2 - a, 1, n - 1).sub_(torch.diff(phi, dim=2 - a) * self.along(self.ax[a].t['inv_sp'][1:n], a))
            self.no_flow(v, a)
            u.append(v)
        return u, phi

    def cfl(self, u):
        rate = 0.0
        for a in range(3):
            f, n = u[a].abs(), self.ax[a].n
            rate = rate + torch.maximum(f.narrow(2 - a, 0, n), f.narrow(2 - a, 1, n)) / self.along(self.ax[a].width, a)
        return float(rate.max())

    def edge_terms(self, u, a, b, lamb):
        """The edges between axes a < b: the vorticity (du_b/dx_a - du_a/dx_b, times `sign`) weighted, times the
        interpolated velocities, added to the Lamb vector of the faces of a and b."""
        d = 3 - a - b
        ta, tb = self.ax[a].t, self.ax[b].t
        na, nb = self.ax[a].n, self.ax[b].n
        fa, fb = u[a], u[b]                     # fa: faces along a, cells along b; fb the other way round
        on = lambda t, key, ax: self.along(t[key], ax)
        for narrow in (True, False):
            if not narrow and self.s['impulse_order'] != 4:
                continue
            lo, hi = (-1, 0) if narrow else (-2, 1)
            q = '1' if narrow else '3'
            b_lo, b_hi = self.cut(fb, a, lo, lo + na + 1), self.cut(fb, a, hi, hi + na + 1)
            a_lo, a_hi = self.cut(fa, b, lo, lo + nb + 1), self.cut(fa, b, hi, hi + nb + 1)
            inv = 'inv_sp' if narrow else 'inv3'
            if narrow:
                weight = on(ta, 'ok', a) * on(tb, 'ok', b)
                if self.s['impulse_order'] == 4:
                    weight = weight * (1 + on(ta, 'l1', a) * on(tb, 'l1', b) / 8)
            else:
                weight = -(on(ta, 'l3', a) * on(tb, 'l3', b)) / 8
            omega = weight * ((b_hi - b_lo) * on(ta, inv, a) - (a_hi - a_lo) * on(tb, inv, b))
            to_a = omega * (on(ta, 'lo' + q, a) * b_lo + on(ta, 'hi' + q, a) * b_hi)
            to_b = omega * (on(tb, 'lo' + q, b) * a_lo + on(tb, 'hi' + q, b) * a_hi)
            for term, ax, n_other, other, sign in ((to_a, a, nb, b, 1.0), (to_b, b, na, a, -1.0)):
                # a face takes the edges at its cell's two ends along the other axis (narrow), or one further out
                if narrow:
                    both = term.narrow(2 - other, 0, n_other) + term.narrow(2 - other, 1, n_other)
                    lamb[ax] += sign * 0.5 * both
                else:
                    c3 = on(self.ax[ax].t, 'c3', ax)
                    lamb[ax].narrow(2 - other, 0, n_other - 1).add_(
                        sign * (c3 * term).narrow(2 - other, 2, n_other - 1))
                    lamb[ax].narrow(2 - other, 1, n_other - 1).add_(
                        sign * (c3 * term).narrow(2 - other, 0, n_other - 1))

    def sweep(self, u, m, base, a0, b, dt, lid_speed):
        lamb = [torch.zeros_like(f) for f in u]
        self.edge_terms(u, 0, 1, lamb)
        self.edge_terms(u, 0, 2, lamb)
        self.edge_terms(u, 1, 2, lamb)
        k = 0.0
        for a in range(3):
            p, n = u[a] * m[a], self.ax[a].n
            k = k + 0.5 * (p.narrow(2 - a, 0, n) + p.narrow(2 - a, 1, n))
        new = []
        for a in range(3):
            n = self.ax[a].n
            inside = slice(1, n)
            cut = lambda f: f.narrow(2 - a, 1, n - 1)
            change = cut(lamb[a]) - torch.diff(k, dim=2 - a) * self.along(self.ax[a].t['inv_sp'][inside], a)
            cc = cut(m[a])
            grad = torch.diff(m[a], dim=2 - a) / self.along(self.ax[a].width, a)
            lap = torch.diff(grad, dim=2 - a) * self.along(self.ax[a].t['inv_sp'][inside], a)
            for t in range(3):
                if t == a:
                    continue
                nt, inv = self.ax[t].n, self.ax[t].t['inv_sp']
                flux = torch.diff(cc, dim=2 - t) * self.along(inv[1:nt], t)
                wall = cut(u[a])
                low = wall.narrow(2 - t, 0, 1) * inv[0]
                high = -wall.narrow(2 - t, nt - 1, 1) * inv[nt]
                if t == 1 and a == 0:
                    high = high + (lid_speed * self.lid[:, 1:n]).unsqueeze(1) * inv[nt]
                lap = lap + torch.diff(torch.cat([low, flux, high], dim=2 - t), dim=2 - t) / self.along(self.ax[t].width, t)
            val = cc + dt * (self.s['nu'] * lap + change)
            f = torch.zeros_like(m[a])
            cut(f).copy_(val if a0 == 0.0 else a0 * cut(base[a]) + b * val)
            new.append(f)
        return new

    def step(self):
        s = self.s
        rates = (float(np.float32(self.rate)), self.viscous)
        use = self.prev if s['dt_lag'] and self.prev else rates
        self.prev = rates
        dt = s['dt_fixed']
        if s['adaptive_dt']:
            dt = min(s['dt_max'], s['cfl_target'] / max(use[0], 1e-300), s['diffusion_limit'] / max(use[1], 1e-300))
        if s['dt_lag'] and self.dt > 0:
            dt = min(dt, 1.1 * self.dt)
        r = s['reinit_r']
        m0 = [r * m + (1 - r) * u for m, u in zip(self.m, self.u)]
        m, u = m0, self.u
        for a0, b in ((0.0, 1.0), (0.75, 0.25), (1 / 3, 2 / 3)):
            m = self.sweep(u, m, m0, a0, b, dt, s['u_lid'])
            u, self.phi = self.project(m)
        self.m, self.u, self.dt, self.rate = m, u, dt, self.cfl(u)
        self.time += dt
        self.count += 1

    def centred(self, a):
        n = self.ax[a].n
        return 0.5 * (self.u[a].narrow(2 - a, 0, n) + self.u[a].narrow(2 - a, 1, n))

    def probes(self):
        out = []
        u, v = self.centred(0), self.centred(1)
        z = self.ax[2].n // 2
        for px, py in PROBES:
            at = [min(a.n - 1, max(0, int(np.searchsorted(a.face, p * 1.0, side='right')) - 1))
                  for a, p in zip(self.ax, (px, py))]
            out += [float(u[z, at[1], at[0]]), float(v[z, at[1], at[0]])]
        return out

    def statistics(self):
        nz, k2 = self.ax[2].n, self.ax[2].n // 2
        k1 = k2 if nz % 2 else k2 - 1
        u, v, w = (0.5 * (f[k1] + f[k2]) for f in (self.centred(0), self.centred(1), self.centred(2)))
        self.sums += self.dt * torch.stack([u, v, u * u, v * v, w * w, u * v])
        h = self.ax[0].n // 2
        cu, cw = (0.5 * (f[:, h - 1] + f[:, h]) for f in (u, w))
        cv = 0.5 * (v[h - 1] + v[h])
        return torch.stack([cu, cv, cu * cu, cv * cv, cw * cw]).cpu().numpy()


def min_pair(sp):
    return np.minimum(sp[:-1], sp[1:])


def exact(c, seed):
    device = 'cuda' if torch.cuda.is_available() else 'cpu'
    runs, probes, lines, dts = [], [], [], []
    for k, s in enumerate(members(c)):
        e = Exact(s, initial_noise(s, seed * 64 + k), device)
        for _ in range(c['steps']):
            e.step()
            if c['kind'] in ('interactive', 'queued'):
                dts.append(e.dt)
                probes.append(e.probes())
                if c['stats']:
                    lines.append(e.statistics())
        runs.append(e)
        if c['count'] > 1:
            e.ax = e.area = e.inv_lam = e.lid = e.sums = None
    if c['kind'] in ('slots', 'ensemble'):
        width = 4 if c['precision'] == 'mixed' else 8
        up = lambda n: (width * n + 255) // 256 * 256 // width
        flat = lambda e: torch.cat([torch.nn.functional.pad(f.reshape(-1), (0, up(f.numel()) - f.numel()))
                                    for f in e.u + e.m])
        return dict(dt=np.array([e.dt for e in runs]), time=np.array([e.time for e in runs]), steps=None,
                    fields=[flat(e) for e in runs], phi=[e.phi for e in runs])
    e = runs[0]
    out = dict(zip(FIELDS, e.u + e.m), phi=e.phi, time=e.time, steps=None, probes=np.array(probes))
    if c['kind'] == 'interactive':
        out['dt'] = np.array(dts)
        if c['stats']:
            out['lines'] = np.array(lines)
    if c['stats']:
        out['sums'] = e.sums.reshape(-1)
    return out
