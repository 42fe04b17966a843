"""What a user of this framework has it do, as measurable cases.

A case is a dict of plain values; ``prepare`` makes what a program holds before the call (the
flow case with its developed or perturbed state, the network with its weights, the snapshots),
``run`` is one pass through the public entry points, ``work`` counts the bytes and operations
the pass cannot do without, and ``exact`` gives the outputs in 64-bit torch or numpy where the
path has a short plain formulation.  Kinds:

``flow``      MAC_CylinderFlow(boundary='ghost_cell', time_scheme='ab2_cn').solve: the main
              path, in plain FP64 and in the FP32 mode, direct or GMRES pressure
``batch``     CylinderBatch.solve: a parameter sweep, many cases a GPU
``cutcell``   MAC_CylinderFlow(boundary='cut_cell', time_scheme='ab2_cn').solve from rest
``legacy``    the time_scheme='legacy' loops: staircase, ghost_cell and cut_cell boundaries
``vortex``    TaylorGreen.step: the periodic verification run
``train``     one training pass of the learned preconditioner: forward and backward
``pod``       SnapshotPOD.fit on wake snapshots held on the GPU
"""
from __future__ import annotations

import importlib
import importlib.util
import math
import os
import sys
from pathlib import Path

import numpy as np
import torch

# a sweep's graph runs many independent chains; a program that steps batches opens the
# runtime's maximum of hardware queues before the CUDA context exists, as bench.py does
os.environ.setdefault('CUDA_DEVICE_MAX_CONNECTIONS', '32')


def _load(name='cfd_cylinder_flow_ghost_cell_gb300'):
    """The package beside this folder (its directory name has dashes) under an importable name."""
    if name not in sys.modules:
        root = Path(__file__).resolve().parents[1] / 'cfd-cylinder-flow-ghost-cell_gb300'
        spec = importlib.util.spec_from_file_location(name, root / '__init__.py', submodule_search_locations=[str(root)])
        sys.modules[name] = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(sys.modules[name])
    return sys.modules[name], importlib.import_module(name + '.modal')


_pkg, _modal = _load()


def listed():
    return [
        # the smallest grid of the tests: a quick look or a unit study, bound by launches and latency
        dict(name='ghost_fp64_96x48', kind='flow', nx=96, ny=48, h=0.1, re=40.0, precision='fp64', pressure='direct',
             extension='neumann', interpolation='bilinear', inflow='uniform', steps=40),
        # the ordinary channel case (20D x 10D, Re 40) in the reference's own precision
        dict(name='ghost_fp64_400x200', kind='flow', nx=400, ny=200, h=0.05, re=40.0, precision='fp64',
             pressure='direct', extension='neumann', interpolation='bilinear', inflow='parabolic', steps=20),
        # the largest single case of the benchmark (40D x 41D), plain FP64: long wake runs
        dict(name='ghost_fp64_800x820', kind='flow', nx=800, ny=820, h=0.05, re=100.0, precision='fp64',
             pressure='direct', extension='neumann', interpolation='bilinear', inflow='uniform', steps=20),
        # the same flow in the FP32 mode, the benchmark's default
        dict(name='ghost_fp32_800x820', kind='flow', nx=800, ny=820, h=0.05, re=100.0, precision='fp32',
             pressure='direct', extension='neumann', interpolation='bilinear', inflow='uniform', steps=20),
        # the reference's GMRES pressure path in its own precision
        dict(name='ghost_gmres_512x256', kind='flow', nx=512, ny=256, h=0.05, re=100.0, precision='fp64',
             pressure='iterative', extension='neumann', interpolation='bilinear', inflow='uniform', steps=4),
        # a parameter sweep in Re, D and position over the benchmark's three grids
        dict(name='sweep_fp32_12', kind='batch', cases=12, precision='fp32', grid_seed=0, steps=10),
        # the embedded-boundary path at the sweep's widest grid, from the projected start
        dict(name='cutcell_800x410', kind='cutcell', nx=800, ny=410, h=0.05, re=100.0, inflow='uniform', slip=False,
             steps=12),
        # the reference's legacy staircase loop on a ragged grid (350 = 2 5 5 7, odd rows)
        dict(name='staircase_350x213', kind='legacy', boundary='staircase', nx=350, ny=213, h=0.06, re=80.0,
             transport='centered', inflow='uniform', steps=40),
        # the verification run at its benchmark size, FP64
        dict(name='vortex_fp64_1024', kind='vortex', n=1024, nu=0.01, dt=1e-3, precision='fp64', steps=20),
        # the same at a coarse, not power-of-two size in the FP32 mode: order-of-accuracy studies
        dict(name='vortex_fp32_250', kind='vortex', n=250, nu=0.01, dt=2e-3, precision='fp32', steps=20),
        # one training pass of the preconditioner network at its benchmark grid and batch
        dict(name='train_4x512x1024', kind='train', batch=4, height=512, width=1024),
        # modal analysis of a recorded wake
        dict(name='pod_96x400x200', kind='pod', snapshots=96, nx=400, ny=200, modes=10),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _smooth_even(m):
    """An even row length whose factors the row transforms take (none above 61)."""
    m = max(8, m + m % 2)
    while True:
        k, f = m, 2
        while f * f <= k:
            if k % f:
                f += 1
            else:
                k //= f
        if k <= 61:
            return m
        m += 2


def draw(rng):
    """Cell Reynolds numbers U h / nu stay at 5 and below: a run goes on from pass to pass, and the
    centred schemes lose their stability on grids much coarser than that."""
    kind = rng.choice(('flow', 'flow', 'flow', 'flow', 'batch', 'cutcell', 'legacy', 'vortex', 'train', 'pod'))
    if kind == 'flow':
        pressure = 'iterative' if rng.random() < 0.2 else 'direct'
        nx = _smooth_even(_log_int(rng, 96, 512 if pressure == 'iterative' else 800))
        ny = max(48, min(820, int(nx * rng.uniform(0.5, 1.02))))
        h = round(rng.uniform(0.045, 0.1) if nx > 200 else rng.uniform(0.08, 0.1), 4)
        return dict(kind=kind, nx=nx, ny=ny if pressure == 'direct' else min(ny, 256), h=h,
                    re=round(rng.uniform(0.4, 1.0) * 5.0 / h, 2), precision=rng.choice(('fp64', 'fp32')), pressure=pressure,
                    extension=rng.choice(('neumann', 'neumann', 'quadratic')),
                    interpolation=rng.choice(('bilinear', 'bilinear', 'biquadratic')),
                    inflow=rng.choice(('uniform', 'parabolic')), steps=4 if pressure == 'iterative' else 20)
    if kind == 'batch':
        return dict(kind=kind, cases=rng.randint(2, 12), precision=rng.choice(('fp64', 'fp32')),
                    grid_seed=rng.randrange(1, 1 << 20), steps=rng.randint(4, 10))
    if kind == 'cutcell':
        nx = _smooth_even(_log_int(rng, 96, 800))
        return dict(kind=kind, nx=nx, ny=max(48, int(nx * rng.uniform(0.4, 0.51))), h=0.1 if nx < 200 else 0.05,
                    re=round(rng.uniform(0.4, 1.0) * (50 if nx < 200 else 100), 2),
                    inflow=rng.choice(('uniform', 'parabolic')), slip=rng.random() < 0.25, steps=12)
    if kind == 'legacy':
        nx = _smooth_even(_log_int(rng, 96, 800))
        return dict(kind=kind, boundary=rng.choice(('staircase', 'ghost_cell', 'cut_cell')), nx=nx,
                    ny=max(48, int(nx * rng.uniform(0.4, 0.61))), h=0.1 if nx < 200 else 0.06,
                    re=round(rng.uniform(0.4, 1.0) * (50 if nx < 200 else 80), 2), transport=rng.choice(('centered', 'upwind')),
                    inflow=rng.choice(('uniform', 'parabolic')), steps=rng.randint(10, 40))
    if kind == 'vortex':
        n = _smooth_even(_log_int(rng, 64, 1020))
        if rng.random() < 0.3:
            n = rng.choice((63, 75, 105, 135, 189, 225, 315, 375, 525, 675, 945))
        return dict(kind=kind, n=n, nu=round(rng.uniform(0.005, 0.1), 4), dt=1e-3 if n > 400 else 2e-3,
                    precision=rng.choice(('fp64', 'fp32')), steps=rng.randint(5, 20))
    if kind == 'train':
        h, w = 8 * _log_int(rng, 6, 64), 8 * _log_int(rng, 12, 128)
        return dict(kind=kind, batch=rng.randint(1, 4), height=h, width=w)
    nx, ny = _log_int(rng, 80, 400), _log_int(rng, 40, 200)
    return dict(kind=kind, snapshots=rng.randint(12, 96), nx=nx, ny=ny, modes=rng.randint(2, 10))


# -- flow cases -----------------------------------------------------------------------------------

DT = 0.002


def _flow_kwargs(c):
    lx, ly = c['nx'] * c['h'], c['ny'] * c['h']
    return dict(nx=c['nx'], ny=c['ny'], Lx=lx, Ly=ly, D=1.0, xc=lx / 4, yc=ly / 2, nu=1.0 / c['re'], verbose=False)


def _perturb(s, integrator, seed, amplitude):
    """Seeded Gaussian noise on the active faces, as the benchmark starts its runs."""
    q = integrator.pack(s.u, s.v)
    q += amplitude * np.random.default_rng(seed).standard_normal(q.size)
    u, v = integrator.unpack(q)
    s.u[:], s.v[:] = u, v


_quiet = dict(dt=DT, perturb_transient=False, save_artifacts=False, verbose=False)


class _Flow:
    """A run under way: the start-up step and two steps are behind it; each pass goes on."""

    def __init__(self, c, seed):
        self.steps = c['steps']
        self.s = _pkg.MAC_CylinderFlow(boundary='ghost_cell', time_scheme='ab2_cn', precision=c['precision'],
                                       pressure_solver=c['pressure'], inflow=c['inflow'],
                                       ghost_pressure_extension=c['extension'],
                                       ghost_velocity_interpolation=c['interpolation'], **_flow_kwargs(c))
        _perturb(self.s, self.s.gg, seed, 1e-3)
        self.s.solve(n_steps=3, **_quiet)

    def run(self):
        s = self.s
        t, cd, cl = s.solve(n_steps=self.steps, **_quiet)
        return dict(u=s.u, v=s.v, p=s.p, forces=np.stack((cd, cl)))


class _Batch:
    """Seeded draws of a sweep; every case is stepped together, from host states and back."""

    def __init__(self, c, seed):
        self.steps = c['steps']
        rng, cases = np.random.default_rng(c['grid_seed']), []
        while len(cases) < c['cases']:
            nx, ny = ((256, 128), (400, 200), (800, 410))[int(rng.integers(3))]
            re, d = rng.uniform(40.0, 100.0), rng.uniform(0.8, 1.2)
            lx, ly = nx * 0.05, ny * 0.05
            xc, yc = lx / 4 + rng.uniform(-0.5, 0.5) * d, ly / 2 + rng.uniform(-0.5, 0.5) * d
            try:
                s = _pkg.MAC_CylinderFlow(boundary='ghost_cell', time_scheme='ab2_cn', precision=c['precision'],
                                          nx=nx, ny=ny, Lx=lx, Ly=ly, D=d, xc=xc, yc=yc, nu=d / re, verbose=False)
            except ValueError:  # a draw whose probes leave the grid
                continue
            _perturb(s, s.gg, seed * 1000 + len(cases), 1e-3)
            cases.append(s)
        self.b = _pkg.CylinderBatch(cases)
        self.b.solve(3, dt=DT)

    def run(self):
        series = self.b.solve(self.steps, dt=DT)
        return [dict(u=s.u, v=s.v, p=s.p, forces=np.stack(r[1:])) for s, r in zip(self.b.cases, series)]


class _CutCell:
    """A run from the projected, perturbed start: every pass begins there, start-up step included."""

    def __init__(self, c, seed):
        self.steps = c['steps']
        self.s = _pkg.MAC_CylinderFlow(boundary='cut_cell', time_scheme='ab2_cn', inflow=c['inflow'],
                                       slip_walls=c['slip'], **_flow_kwargs(c))
        _perturb(self.s, self.s.cc, seed, 1e-3)
        self.first = self.s.u.copy(), self.s.v.copy(), self.s.p.copy()

    def run(self):
        s = self.s
        for field, start in zip((s.u, s.v, s.p), self.first):
            field[...] = start
        s.time = 0.0
        s.cc.set_history(None, None, None)
        t, cd, cl = s.solve(n_steps=self.steps, **_quiet)
        return dict(u=s.u, v=s.v, p=s.p, forces=np.stack((cd, cl)))


class _Legacy:
    """The legacy loops, under way from a perturbed field; each pass goes on."""

    def __init__(self, c, seed):
        self.steps = c['steps']
        self.s = s = _pkg.MAC_CylinderFlow(boundary=c['boundary'], time_scheme='legacy', transport=c['transport'],
                                           inflow=c['inflow'], **_flow_kwargs(c))
        rng = np.random.default_rng(seed)
        s.v[1:-1] += 1e-3 * rng.standard_normal(s.v[1:-1].shape) * (s.v[1:-1] == 0) * ~(s.mask[1:] | s.mask[:-1])
        s.solve(n_steps=3, **_quiet)

    def run(self):
        s = self.s
        t, cd, cl = s.solve(n_steps=self.steps, **_quiet)
        return dict(u=s.u, v=s.v, p=s.p, forces=np.stack((cd, cl)))


# -- the periodic vortex --------------------------------------------------------------------------

def _vortex_fields(c, seed):
    """The analytic vortex with a few solenoidal large-scale modes of seeded phase added."""
    n, rng = c['n'], np.random.default_rng(seed)
    q, p = _pkg.taylor_green.exact(n, c['nu'], 0.0)
    x = np.arange(n) * (2 * np.pi / n)
    for k in range(1, 4):  # shear layers u(y) and v(x): free of divergence on the staggered grid
        a, b = rng.uniform(0, 2 * np.pi, 2)
        w = 0.1 / k
        q[:n * n] += np.repeat(w * np.sin(k * (x + np.pi / n) + a), n)
        q[n * n:] += np.tile(w * np.sin(k * (x + np.pi / n) + b), n)
    return q, p


class _Vortex:
    """A whole verification run on a handle: set the field, step, read velocity and pressures."""

    def __init__(self, c, seed):
        self.c = c
        self.case = _pkg.taylor_green.TaylorGreen(c['n'], c['nu'], c['precision'])
        self.q, self.p = _vortex_fields(c, seed)

    def run(self):
        self.case.set_state(self.q, self.p)
        self.case.step(self.c['dt'], self.c['steps'])
        q, half, out = self.case.state()
        return dict(q=q, half=half, out=out)


def _vortex_exact(c, seed):
    n, nu, dt = c['n'], c['nu'], c['dt']
    h = 2 * math.pi / n
    dev = 'cuda' if torch.cuda.is_available() else 'cpu'
    q, p = _vortex_fields(c, seed)
    u, v = (torch.from_numpy(f.reshape(n, n)).to(dev) for f in (q[:n * n], q[n * n:]))
    p = torch.from_numpy(p).to(dev)
    s2 = torch.sin(math.pi * torch.arange(n, device=dev, dtype=torch.float64) / n) ** 2
    lam = -4 * (s2[:, None] + s2[None, :]) / h ** 2
    inv = torch.where(lam == 0, torch.zeros_like(lam), 1 / torch.where(lam == 0, torch.ones_like(lam), lam))
    east, west = (lambda f: f.roll(-1, 1)), (lambda f: f.roll(1, 1))
    north, south = (lambda f: f.roll(-1, 0)), (lambda f: f.roll(1, 0))

    def spectral(f, factor):
        return torch.fft.ifft2(torch.fft.fft2(f) * factor).real

    def advection(u, v):
        ue, uw = (u + east(u)) / 2, (west(u) + u) / 2
        au = -((ue * ue - uw * uw) + ((west(north(v)) + north(v)) / 2 * (u + north(u)) / 2
                                      - (west(v) + v) / 2 * (south(u) + u) / 2)) / h
        vn, vs = (v + north(v)) / 2, (south(v) + v) / 2
        av = -((vn * vn - vs * vs) + ((south(east(u)) + east(u)) / 2 * (v + east(v)) / 2
                                      - (south(u) + u) / 2 * (west(v) + v) / 2)) / h
        return au, av

    def lap(f):
        return nu * ((east(f) - f) - (f - west(f)) + (north(f) - f) - (f - south(f))) / h ** 2

    def grad(f):
        return (f - west(f)) / h, (f - south(f)) / h

    def project(u, v, step):
        phi = spectral(((east(u) - u) + (north(v) - v)) / h / step, inv)
        gx, gy = grad(phi)
        return u - step * gx, v - step * gy, phi

    prev, out = None, p
    for _ in range(c['steps']):
        au, av = advection(u, v)
        gx, gy = grad(p)
        if prev is None:
            hu, hv, _ = project(u + dt / 2 * (au + lap(u) - gx), v + dt / 2 * (av + lap(v) - gy), dt / 2)
            eu, ev = advection(hu, hv)
        else:
            eu, ev = 1.5 * au - 0.5 * prev[0], 1.5 * av - 0.5 * prev[1]
        ru, rv = u + dt * (eu + lap(u) / 2 - gx), v + dt * (ev + lap(v) / 2 - gy)
        cn = 1 / (1 - dt / 2 * nu * lam)
        un, vn, _ = project(spectral(ru, cn), spectral(rv, cn), dt)
        du, dv = ru - (un - dt / 2 * lap(un)), rv - (vn - dt / 2 * lap(vn))
        _, _, inc = project(un + du, vn + dv, dt)
        p = p + inc
        out = p + (1.0 if prev is None else 0.5) * inc
        u, v, prev = un, vn, (au, av)
    return dict(q=torch.cat((u.reshape(-1), v.reshape(-1))).cpu().numpy(), half=p.cpu().numpy(), out=out.cpu().numpy())


# -- the learned preconditioner -------------------------------------------------------------------

class _Train:
    """One training pass: the network's output, the masked loss and every parameter's gradient."""

    def __init__(self, c, seed):
        b, hh, ww = c['batch'], c['height'], c['width']
        self.net = _pkg.learned.UNet(b, hh, ww)
        self.weights = _pkg.learned.UNetWeights()
        self.weights.load(_train_weights(seed))
        self.x, self.y, self.mask = _train_data(c, seed)

    def run(self):
        params = self.weights.parameters()
        for p in params:
            p.grad = None
        pred = _pkg.learned.apply(self.net, self.weights, self.x)
        loss = (((pred - self.y) * self.mask) ** 2).sum() / (self.mask.sum() * self.x.shape[0])
        loss.backward()
        return dict(pred=pred.detach(), loss=loss.detach(), grads=[p.grad for p in params])


_LAYERS = ((2, 16, 0), (16, 16, 0), (16, 32, 1), (32, 32, 1), (32, 64, 2), (64, 64, 2), (64, 64, 3), (64, 64, 3),
           (128, 64, 2), (96, 32, 1), (48, 16, 0), (16, 1, 0))  # channels in, channels out, level


def _train_weights(seed):
    """Weights of a network in training: scaled normal, with small biases."""
    rng, state = np.random.default_rng(seed), {}
    for k, (i, o, _) in enumerate(_LAYERS):
        state[f'w{k}'] = (rng.standard_normal((o, i, 3, 3)) * (2 / (9 * i)) ** 0.5).astype(np.float32)
        state[f'b{k}'] = (rng.standard_normal(o) * 0.02).astype(np.float32)
    return state


def _train_data(c, seed):
    """Normalised right-hand sides with a solid disc, and smooth corrections as targets."""
    b, hh, ww = c['batch'], c['height'], c['width']
    g = torch.Generator(device='cuda').manual_seed(seed)
    yy = torch.arange(hh, device='cuda', dtype=torch.float32)[:, None]
    xx = torch.arange(ww, device='cuda', dtype=torch.float32)[None, :]
    mask = ((yy - hh / 2) ** 2 + (xx - ww / 5) ** 2 > (hh / 20) ** 2).float()
    rhs = torch.randn(b, hh, ww, device='cuda', generator=g) * mask
    rhs = rhs / rhs.abs().amax(dim=(1, 2), keepdim=True)
    x = torch.stack((rhs, mask.expand(b, hh, ww)), dim=1).contiguous()
    a = torch.rand(b, 1, 1, 1, device='cuda', generator=g)
    y = 0.1 * torch.sin(6.28 * (xx / ww + a)) * torch.cos(6.28 * (yy / hh - a)) * mask
    return x, y.contiguous(), mask


def _train_exact(c, seed):
    x, y, mask = (t.double() for t in _train_data(c, seed))
    state = _train_weights(seed)
    # the network reads its FP32 master weights as BF16
    w = [torch.from_numpy(state[f'w{k}']).to(torch.bfloat16).double().cuda().requires_grad_() for k in range(12)]
    b = [torch.from_numpy(state[f'b{k}']).double().cuda().requires_grad_() for k in range(12)]
    f = torch.nn.functional

    def conv(k, t):
        return f.conv2d(t, w[k], b[k], padding=1)

    e0 = conv(1, conv(0, x).relu()).relu()
    e1 = conv(3, conv(2, f.avg_pool2d(e0, 2)).relu()).relu()
    e2 = conv(5, conv(4, f.avg_pool2d(e1, 2)).relu()).relu()
    d = conv(7, conv(6, f.avg_pool2d(e2, 2)).relu()).relu()
    for k, skip in ((8, e2), (9, e1), (10, e0)):
        d = conv(k, torch.cat((f.interpolate(d, scale_factor=2, mode='nearest'), skip), dim=1)).relu()
    pred = conv(11, d)
    loss = (((pred - y) * mask) ** 2).sum() / (mask.sum() * x.shape[0])
    grads = torch.autograd.grad(loss, w + b)
    return dict(pred=pred.detach(), loss=loss.detach(), grads=list(grads))


# -- modal analysis -------------------------------------------------------------------------------

def _snapshots(c, seed):
    """A convecting wake: travelling wave pairs of decaying energy over a mean, with weak noise."""
    m, nx, ny = c['snapshots'], c['nx'], c['ny']
    g = torch.Generator(device='cuda').manual_seed(seed)
    f64 = dict(dtype=torch.float64, device='cuda')
    t = torch.arange(m, **f64)[:, None, None] * (6.283185307 / m)
    y = torch.linspace(-1, 1, ny, **f64)[None, :, None]
    x = torch.linspace(0, 1, nx, **f64)[None, None, :]
    snaps = (1 - torch.exp(-4 * y * y)).expand(m, ny, nx).clone()
    for k in range(1, 7):
        a, b = torch.rand(2, **f64, generator=g)
        snaps += 0.6 ** k * torch.exp(-(k + 1) * y * y) * (torch.sin(k * (6.28 * x - t) + 6.28 * a)
                                                         + 0.4 * b * torch.cos(k * t))
    return snaps + 1e-5 * torch.randn(m, ny, nx, **f64, generator=g)


class _Pod:
    def __init__(self, c, seed):
        self.modes, self.x = c['modes'], _snapshots(c, seed)

    def run(self):
        p = _modal.SnapshotPOD(self.modes).fit(self.x)
        # the singular values are the square roots of these energies times the snapshot count; that
        # of the null mode of mean-free snapshots is the root of a rounding error
        return dict(mean=p.mean_field, energies=p.modal_energies, ratios=p.energy_ratios,
                    cumulative=p.cumulative_energy, modes=p.spatial_modes, coefficients=p.temporal_coeffs)


def _pod_exact(c, seed):
    x = _snapshots(c, seed).cpu().numpy().reshape(c['snapshots'], -1)
    m = x.shape[0]
    mean = x.mean(axis=0)
    d = x - mean
    lam, vec = np.linalg.eigh(d @ d.T / m)
    lam, vec = np.maximum(lam[::-1], 0.0), vec[:, ::-1]
    # the sign of an eigenvector is a convention: its values have none to compare with
    return dict(mean=mean.reshape(c['ny'], c['nx']), energies=lam, ratios=lam / lam.sum(),
                cumulative=np.cumsum(lam / lam.sum()), modes=None, coefficients=None)


# -- the interface --------------------------------------------------------------------------------

_KINDS = dict(flow=_Flow, batch=_Batch, cutcell=_CutCell, legacy=_Legacy, vortex=_Vortex, train=_Train, pod=_Pod)


def prepare(case, seed):
    return _KINDS[case['kind']](case, seed)


def run(state):
    return state.run()


def exact(case, seed):
    """The flow paths are whole solvers (geometry, ghost or cut-cell operators, boundary
    corrections): no short plain form, so None."""
    if case['kind'] == 'vortex':
        return _vortex_exact(case, seed)
    if case['kind'] == 'train':
        return _train_exact(case, seed)
    if case['kind'] == 'pod':
        return _pod_exact(case, seed)
    return None


def _flow_work(cells, nx, steps, solves):
    """Per step: u, v, p and the AB2 history (u, v) read and written once in FP64; each solve two
    real row transforms of 2.5 log2(nx) operations a point and a tridiagonal column solve, and
    some 120 operations a cell for the momentum terms, the projections and the residuals."""
    return dict(bytes=80 * cells * steps, flops=cells * steps * (solves * (5 * math.log2(nx) + 8) + 120))


def work(case):
    c = case
    if c['kind'] == 'flow':
        # two momentum and two pressure solves a step; GMRES: about 18 inverses a pressure solve
        return _flow_work(c['nx'] * c['ny'], c['nx'], c['steps'], 4 if c['pressure'] == 'direct' else 38)
    if c['kind'] == 'batch':
        cells = c['cases'] * (256 * 128 + 400 * 200 + 800 * 410) // 3
        return _flow_work(cells, 400, c['steps'], 4)
    if c['kind'] == 'cutcell':
        # two pressure solves and about five GMRES products of 100 operations a step
        w = _flow_work(c['nx'] * c['ny'], c['nx'], c['steps'], 2)
        return dict(bytes=w['bytes'], flops=w['flops'] + 500 * c['nx'] * c['ny'] * c['steps'])
    if c['kind'] == 'legacy':
        return _flow_work(c['nx'] * c['ny'], c['nx'], c['steps'], 1)
    if c['kind'] == 'vortex':
        # per step two projections and one two-component Helmholtz solve, each field a forward
        # and an inverse real 2-D transform; fields as in the flow cases
        n = c['n']
        return dict(bytes=80 * n * n * c['steps'], flops=n * n * c['steps'] * (4 * 10 * math.log2(n) + 120))
    if c['kind'] == 'train':
        pix, b = c['height'] * c['width'], c['batch']
        # forward, weight gradient and (but for the first layer) data gradient
        flops = sum((3 if k else 2) * 18 * i * o * pix / 4 ** lv for k, (i, o, lv) in enumerate(_LAYERS)) * b
        # every activation written and read once in each direction
        acts = sum(o * pix / 4 ** lv for _, o, lv in _LAYERS) * b
        return dict(bytes=4 * acts * 4, flops=flops)
    m, n, k = c['snapshots'], c['nx'] * c['ny'], c['modes']
    return dict(bytes=8 * n * (m + k + 1), flops=n * (m * (m + 1) + 4 * m * k + 2 * m))
