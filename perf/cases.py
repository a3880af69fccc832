"""Performance cases of the framework: what is timed, on which inputs, and the
values a plain 64-bit evaluation gives.

A case is a dict of plain values.  ``kind`` says which use it stands for:

* ``forward``: a forecast that stays on the device.  New initial fields go in
  (``Dycore.upload_device``), the model takes ``steps`` steps with the vertical
  remap every ``remap_every`` (``Dycore.step``, with its stability check, as the
  time loop calls it), and the prognostic fields come out
  (``Dycore.download_device``).  ``form`` is the FP64 or the mixed form.
* ``gradient``: a differentiated forecast through ``atmdyn.adjoint.integrate``
  with checkpoints, the loss being the sum of squares of the final potential
  temperature, over the whole domain (``radius`` 0) or under a Gaussian mask
  of ``radius`` metres; returns the loss and the four gradients.
* ``physics``: ``atmdyn.model.run_model`` with radiation and column physics.
* ``ensemble``: independent members of uneven sizes advanced by one CUDA graph.

Grids, layer counts, time steps and remap intervals are those of
``atmdyn.ic.config``, ``atmdyn.ic.ensemble_members`` and the tests.  Fields are
the jet and bubble states of ``atmdyn.ic`` (formed here on the GPU), with smooth
noise on every field, as a forecast meets them after its first steps.
"""
import math
import os
import random
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for _p in (os.path.join(os.getcwd(), 'atmosphere-model_b200'), os.path.join(ROOT, 'atmosphere-model_b200')):
    if os.path.isdir(_p):
        if _p not in sys.path:
            sys.path.insert(0, _p)
        break

from atmdyn import gas_optics, ic, model  # noqa: E402
from atmdyn.adjoint import CUDA_STREAM_LEGACY, gaussian_mask, integrate  # noqa: E402
from atmdyn.dycore import Dycore, with_halo  # noqa: E402
from atmdyn.ensemble import Ensemble  # noqa: E402

FIELDS = ('dp', 'pt', 'ud', 'vd')
# an exact evaluation runs one torch operation at a time: its budget in
# cell-steps (forward) and in cells x steps kept for autograd (gradient)
EXACT_FORWARD, EXACT_GRADIENT = 6.0e8, 1.0e6


def _forward(name, form, state, nx, ny, nlay, steps, remap_every):
    return dict(name=name, kind='forward', form=form, state=state, nx=nx, ny=ny, nlay=nlay, steps=steps,
                remap_every=remap_every)


def _gradient(name, nx, ny, nlay, steps, checkpoint_every, radius):
    return dict(name=name, kind='gradient', state='jet', nx=nx, ny=ny, nlay=nlay, steps=steps, remap_every=5,
                checkpoint_every=checkpoint_every, radius=radius)


def listed():
    return [
        # the smallest ensemble member on its own: a step is a dozen launches of a few microseconds each
        _forward('fp64_64x64x20', 'fp64', 'bubble', 64, 64, 20, 5, 5),
        # the parity configuration: 128 x 128 x 20 bubble, remap every 5
        _forward('fp64_128x128x20', 'fp64', 'bubble', 128, 128, 20, 5, 5),
        # a regional grid with no convenient factor in any direction
        _forward('fp64_251x187x27', 'fp64', 'jet', 251, 187, 27, 4, 4),
        # the headline grid over one remap interval
        _forward('fp64_1024x1024x64', 'fp64', 'jet', 1024, 1024, 64, 8, 8),
        # the mixed form on a small ragged grid, and on the headline grid
        _forward('mixed_150x130x48', 'mixed', 'jet', 150, 130, 48, 5, 5),
        _forward('mixed_1024x1024x64', 'mixed', 'jet', 1024, 1024, 64, 8, 8),
        # sensitivities of a small domain, where latency counts
        _gradient('gradient_64x64x20', 64, 64, 20, 5, 5, 0.0),
        # the differentiation grid, every column carrying an adjoint: one checkpoint segment
        _gradient('gradient_512x512x32', 512, 512, 32, 5, 5, 0.0),
        # a longer trajectory (recomputed segments) with a regional loss
        _gradient('gradient_301x203x40_masked', 301, 203, 40, 10, 5, 1.5e6),
        # the model's whole time loop with radiation at its first step
        dict(name='physics_192x160x48', kind='physics', form='fp64', state='bubble', nx=192, ny=160, nlay=48,
             steps=2, remap_every=2),
        # eight members of uneven sizes over one remap cycle
        dict(name='ensemble_8_members', kind='ensemble', form='mixed', members=8, mix=3, steps=5, remap_every=5),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['forward', 'forward', 'forward', 'gradient', 'gradient', 'physics', 'ensemble'])
    state = rng.choice(['jet', 'bubble'])
    if kind == 'ensemble':
        return dict(kind=kind, form='mixed', members=rng.randint(4, 10), mix=rng.randint(0, 10 ** 6), steps=5,
                    remap_every=5)
    top = {'forward': 1024, 'gradient': 512, 'physics': 320}[kind]
    nx, ny = _log_int(rng, 48, top), _log_int(rng, 48, top)
    nlay = rng.randint(12, 64)
    if kind == 'gradient':
        nlay = min(nlay, max(12, 8400000 // (nx * ny)))
        steps = rng.randint(2, 6)
        case = _gradient('', nx, ny, nlay, steps, rng.randint(2, 5), rng.choice([0.0, 0.0, 1.5e6])) | {'state': state}
        del case['name']
        return case
    if kind == 'physics':
        return dict(kind=kind, form=rng.choice(['fp64', 'mixed']), state='bubble', nx=nx, ny=ny, nlay=nlay, steps=2,
                    remap_every=2)
    case = _forward('', rng.choice(['fp64', 'mixed']), state, nx, ny, nlay, rng.randint(3, 8), rng.randint(3, 8))
    del case['name']
    return case


# ---- inputs -----------------------------------------------------------------

def _device():
    return torch.device('cuda' if torch.cuda.is_available() else 'cpu')


def _geometry(state, nx, ny):
    """Cell sizes and time step of the grid: the configurations' domains, at
    this resolution."""
    if state == 'jet':
        return 25e3 * 1024 / nx, 25e3 * 1024 / ny, 30.0 * 1024 / max(nx, ny) / 2
    return 50e3 * 128 / nx, 50e3 * 128 / ny, 60.0 * 128 / max(nx, ny)


def _smooth(gen, shape, rms, dev, cells=3.0):
    """White noise smoothed by a Gaussian of ``cells`` cells, level by level."""
    ny, nx = shape[-2:]
    ky = torch.fft.fftfreq(ny, device=dev, dtype=torch.float64)[:, None]
    kx = torch.fft.rfftfreq(nx, device=dev, dtype=torch.float64)[None, :]
    g = torch.exp(-2.0 * (math.pi * cells) ** 2 * (kx * kx + ky * ky))
    out = torch.empty(shape, dtype=torch.float64, device=dev)
    for k in range(shape[0]):
        a = torch.randn((ny, nx), generator=gen, dtype=torch.float64, device=dev)
        a = torch.fft.irfft2(torch.fft.rfft2(a) * g, s=(ny, nx))
        out[k] = a * (rms / a.std())
    return out


def _fields(state, nx, ny, nlay, seed):
    """(dp, pt, ud, vd, ts) of a jet or bubble state with smooth noise."""
    dev = _device()
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(seed) * 1000003 + 17)
    dx, dy, _ = _geometry(state, nx, ny)
    f64 = dict(dtype=torch.float64, device=dev)
    ptop, p0, kap = 1.0e4, ic.P0, ic.KAPPA
    sig = (nlay - torch.arange(nlay + 1, **f64)) / nlay
    ps = 1.0e5 + _smooth(gen, (1, ny, nx), 30.0, dev)
    lev = ptop + sig[:, None, None] * (ps - ptop)
    pb, pt_ = lev[:-1], lev[1:]
    dp = (pb - pt_).contiguous()
    a = kap - 0.1
    thick = 300.0 / a * ((pb / p0) ** a - (pt_ / p0) ** a)
    pm = 0.5 * (pb + pt_)
    xc = (torch.arange(nx, **f64) + 0.5) * dx
    yc = (torch.arange(ny, **f64) + 0.5) * dy
    lx, ly = nx * dx, ny * dy
    if state == 'jet':
        w, u0 = max(500e3, 4 * dy), 30.0
        lnr = math.log(1.0e5 / ptop)
        ubar = u0 * 2 * w * math.tanh(ly / (2 * w)) / ly
        integ = u0 * w * (torch.tanh((yc - ly / 2) / w) + math.tanh(ly / (2 * w))) - ubar * yc
        dt_y = -1e-4 / (ic.R_DRY * lnr) * integ
        thick = thick + dt_y[None, :, None] * torch.log(pb / pt_)
        yf = torch.arange(ny, **f64) * dy
        prof = u0 / torch.cosh((yf - ly / 2) / w) ** 2 - ubar
        ud = prof[None, :, None] * (torch.log(1.0e5 / pm) / lnr)
        th = torch.zeros((), **f64)
    else:
        r2 = ((xc[None, :] - lx / 2) ** 2 + (yc[:, None] - ly / 2) ** 2) / (500e3) ** 2
        th = 2.0 * torch.exp(-r2)[None] * torch.exp(-((pm - 7.0e4) / 2.0e4) ** 2)
        ud = torch.full((nlay, ny, nx), 10.0, **f64)
    pt = ic.R_DRY * thick / (ic.CP_DRY * (pb ** kap - pt_ ** kap)) + th / p0 ** kap
    pt = pt + _smooth(gen, (nlay, ny, nx), 0.3, dev) / p0 ** kap
    ud = ud + _smooth(gen, (nlay, ny, nx), 0.5, dev)
    vd = _smooth(gen, (nlay, ny, nx), 0.5, dev)
    ts = 288.0 + _smooth(gen, (1, ny, nx), 2.0, dev)[0]
    return dp, pt.contiguous(), ud.contiguous(), vd, ts


def _blank(case, state, nx, ny, nlay):
    """The grid, coordinate and constants a Dycore is made with; its fields
    are those of a resting state, replaced before every forecast."""
    dx, dy, dt = _geometry(state, nx, ny)
    ak, bk = ic.sigma_coordinate(nlay)
    shape = (nlay, ny, nx)
    const = lambda v: np.broadcast_to(np.float64(v), shape)  # noqa: E731
    return ic.InitialState(nx, ny, nlay, dx, dy, ak, bk, const(9.0e4 / nlay), const(11.0), const(0.0), const(0.0),
                           np.zeros((ny, nx)), dt=dt, remap_every=case['remap_every'], ts=np.full((ny, nx), 288.0))


def _on_torch_stream(dyn):
    h = torch.cuda.current_stream().cuda_stream
    dyn.set_stream(h if h else CUDA_STREAM_LEGACY)


def _members(case):
    """(state, n, nlay) of each member: sizes as ic.ensemble_members mixes them."""
    r = random.Random(case['mix'])
    out = []
    for m in range(case['members']):
        n = 512 if m == 0 else r.choice([64, 96, 128, 256])
        out.append((r.choice(['jet', 'bubble']), n, r.choice([20, 32, 48, 64]) if m else 20))
    return out


def prepare(case, seed):
    kind = case['kind']
    if kind == 'ensemble':
        mem = _members(case)
        fields = [_fields(s, n, n, L, seed * 100 + i)[:4] for i, (s, n, L) in enumerate(mem)]
        ens = Ensemble([_blank(case, s, n, n, L) for s, n, L in mem], case['form'], nstreams=8)
        ens.capture(case['remap_every'])
        out = [[torch.empty_like(f) for f in fs] for fs in fields]
        return dict(case=case, ens=ens, fields=fields, out=out)
    nx, ny, nlay = case['nx'], case['ny'], case['nlay']
    fields = _fields(case['state'], nx, ny, nlay, seed)
    st = _blank(case, case['state'], nx, ny, nlay)
    dyn = Dycore(st, case.get('form', 'fp64'))
    _on_torch_stream(dyn)
    s = dict(case=case, dyn=dyn, st=st, dt=st.dt, fields=fields[:4])
    if kind == 'gradient':
        dyn.adj_enable()
        s['mask'] = gaussian_mask(st, case['radius'], fields[0].device) if case['radius'] else None
    else:
        s['out'] = [torch.empty_like(f) for f in fields[:4]]
    if kind == 'physics':
        s['ts'] = with_halo(fields[4].cpu().numpy()[None])
        dyn.set_radiation(gas_optics.synthetic(1))
        n = case['steps']
        s['tc'] = model.TimeControl(dt_max=st.dt, run_duration=st.dt * n, dt_radiation=st.dt * n, dt_physics=st.dt,
                                    dt_remap=st.dt * case['remap_every'])
    return s


def run(s):
    case = s['case']
    kind = case['kind']
    if kind == 'ensemble':
        ens = s['ens']
        for d, fs in zip(ens.dyn, s['fields']):
            for name, t in zip(FIELDS, fs):
                d.upload_device(name, t)
        ens.synchronize()
        ens.replay(1)
        ens.synchronize()
        for d, ts in zip(ens.dyn, s['out']):
            for name, t in zip(FIELDS, ts):
                d.download_device(name, t)
        ens.synchronize()
        return s['out']
    dyn, dt = s['dyn'], s['dt']
    if kind == 'gradient':
        x = [t.detach().requires_grad_() for t in s['fields']]
        out = integrate(dyn, x, case['steps'], dt, case['remap_every'], case['checkpoint_every'])
        th2 = out[1] * out[1]
        loss = (th2 if s['mask'] is None else th2 * s['mask']).sum()
        loss.backward()
        return {'loss': loss.detach(), 'gradients': [t.grad for t in x]}
    for name, t in zip(FIELDS, s['fields']):
        dyn.upload_device(name, t)
    if kind == 'physics':
        dyn.upload('ts', s['ts'])
        res = model.run_model(dyn, s['tc'], physics=True, radiation=True)
        stable, extra = res.stable, [dyn.get('ts')[0]]
    else:
        for n in range(1, case['steps'] + 1):
            stable = dyn.step(dt, remap=n % case['remap_every'] == 0)
        extra = []
    for name, t in zip(FIELDS, s['out']):
        dyn.download_device(name, t)
    return {'fields': s['out'], 'stable': int(stable), 'surface': extra}


def _sizes(case):
    """(cells, columns, cells remapped) of one pass."""
    if case['kind'] == 'ensemble':
        cells = sum(n * n * L for _, n, L in _members(case))
        cols = sum(n * n for _, n, L in _members(case))
    else:
        cells, cols = case['nx'] * case['ny'] * case['nlay'], case['nx'] * case['ny']
    return cells, cols, cells * (case['steps'] // case['remap_every'])


def work(case):
    """One pass's inputs read and outputs written once, and the operations of
    the scheme per cell: about 1700 for a step's sweeps, columns and corner
    interpolation, 600 for a remap, three times both for the reverse of a
    step, 150 for the physics, and 500 per layer and g-point of the radiation."""
    cells, cols, remapped = _sizes(case)
    flops = 1700.0 * cells * case['steps'] + 600.0 * remapped
    if case['kind'] == 'gradient':
        flops *= 4
    if case['kind'] == 'physics':
        flops += 150.0 * cells * case['steps'] + 500.0 * 16 * cells
    return {'bytes': 8.0 * (8 * cells + (2 * cols if case['kind'] == 'physics' else 0)), 'flops': flops}


# ---- the scheme in plain 64-bit torch ----------------------------------------
# Fields are (nlay, ny, nx), periodic in y and x, so the neighbour (x+i, y+j) of
# every point is a roll.  At a kink the derivative is that of the branch taken:
# min and max keep the argument they return.

def _at(f, i, j):
    if i or j:
        f = torch.roll(f, shifts=(-j, -i), dims=(-2, -1))
    return f


def _min(a, b):
    return torch.where(b < a, b, a)


def _max(a, b):
    return torch.where(a < b, b, a)


def _slope(q, i, j):
    qm, qp = _at(q, -i, -j), _at(q, i, j)
    d = (qp - qm) * 0.25
    hi = _max(_max(qp, q), qm) - q
    lo = q - _min(_min(qp, q), qm)
    return torch.copysign(_min(_min(d.abs(), lo), hi), d)


def _edges(q, i, j, kind):
    qm, qp, m = _at(q, -i, -j), _at(q, i, j), _slope(q, i, j)
    left = (qm - q) * 0.5 + (_at(m, -i, -j) - m) / 3
    right = (qp - q) * 0.5 + (m - _at(m, i, j)) / 3
    if kind == 'unconstrained':
        return left, right
    d = (qp - qm) * 0.25
    lim = 2 * d.abs()
    left = -torch.copysign(_min(lim, left.abs()), d)
    right = torch.copysign(_min(lim, right.abs()), d)
    if kind == 'nonnegative':
        left, right = _max(left, -q), _max(right, -q)
        a, b = right - left, -3 * (right + left)
        with torch.no_grad():
            safe = torch.where(b == 0, torch.ones_like(b), b)
            fix = (a.abs() < -b) & (q + a * a / (4 * safe) + b / 12 < 0)
            both = fix & (left * right > 0)
            from_right = fix & ~both & (left > right)
            from_left = fix & ~both & ~from_right
        zero = torch.zeros_like(left)
        l2 = torch.where(both, zero, torch.where(from_right, 2 * right.abs(), left))
        right = torch.where(both, zero, torch.where(from_left, 2 * left.abs(), right))
        left = l2
    return left, right


def _flux(q, c, i, j, kind):
    """Upwind PPM value at the interface between a cell's lower neighbour and the cell."""
    left, right = _edges(q, i, j, kind)
    qm, lm, rm = _at(q, -i, -j), _at(left, -i, -j), _at(right, -i, -j)
    s = c.abs()
    k1, k2 = (1 - 2 * s) * (1 - s), s * (s - 1)
    pos = c > 0
    out = torch.where(pos, qm + k1 * rm + k2 * lm, q + k1 * left + k2 * right)
    if kind == 'constrained':
        flat = (3 * (left + right).abs() > (left - right).abs()) & (3 * (lm + rm).abs() > (lm - rm).abs())
        out = torch.where(flat, torch.where(pos, qm, q), out)
    return out


def _inner(q, c0, c1, den, i, j, ra):
    f0 = torch.where(c0 > 0, _at(q, -i, -j), q)
    f1 = torch.where(c1 > 0, q, _at(q, i, j))
    return 0.5 * (q + den * (q - ra * (f1 - f0)))


class _Scheme:
    def __init__(self, st, dev):
        self.st, self.dev, self.L = st, dev, st.nlay
        self.rdx, self.rdy = 1 / st.dx, 1 / st.dy
        self.ra = 1 / (st.dx * st.dy)
        self.div = (st.divdamp * st.dx * st.dy) ** 2
        vort = st.vortdamp * st.dx * st.dy
        self.vx, self.vy = st.dy * self.rdx * vort, st.dx * self.rdy * vort
        self.ak = torch.tensor(st.ak, device=dev)
        self.bk = torch.tensor(st.bk, device=dev)
        self.ptop = float(st.ak[0])

    def lap(self, q):
        return (-2 * q * (self.rdx ** 2 + self.rdy ** 2) + (_at(q, 1, 0) + _at(q, -1, 0)) * self.rdx ** 2
                + (_at(q, 0, 1) + _at(q, 0, -1)) * self.rdy ** 2)

    def mass(self, dp, pt, uc, vc, dt, kind, heat):
        dtdx, dtdy = dt * self.rdx, dt * self.rdy
        vn, un = _at(vc, 0, 1), _at(uc, 1, 0)
        dy, dx = 1 / (1 - dtdy * (vn - vc)), 1 / (1 - dtdx * (un - uc))
        cx, cy = dtdx * uc, dtdx * vc
        fx, fy, gx, gy = [], [], [], []
        for q in (dp, pt):
            fx.append(_flux(_inner(q, cy, dtdx * vn, dy, 0, 1, self.ra), cx, 1, 0, kind))
            fy.append(_flux(_inner(q, cx, dtdx * un, dx, 1, 0, self.ra), cy, 0, 1, kind))
        mx, my = fx[0] * cx, fy[0] * cy
        ld, lp = self.lap(dp), self.lap(pt)
        new = dp - (_at(mx, 1, 0) - mx + dtdx * self.vx * (_at(ld, 1, 0) - 2 * ld + _at(ld, -1, 0)))
        new = new - (_at(my, 0, 1) - my + dtdy * self.vy * (_at(ld, 0, 1) - 2 * ld + _at(ld, 0, -1)))
        hx = (fx[1] + self.vx * (lp - _at(lp, -1, 0))) * mx
        hy = (fy[1] + self.vy * (lp - _at(lp, 0, -1))) * my
        num = dp * pt - (_at(hx, 1, 0) - hx) - (_at(hy, 0, 1) - hy)
        if heat is not None:
            num = num + dt * dp * heat
        return new, num / new

    def levels(self, dp):
        """Interface pressures, bottom to top."""
        up = torch.flip(torch.cumsum(torch.flip(dp, (0,)), 0), (0,)) + self.ptop
        return torch.cat([up, torch.full_like(dp[:1], self.ptop)])

    def column(self, dp, pt):
        pk = self.levels(dp) ** ic.KAPPA
        z = torch.cumsum(ic.CP_DRY * pt * (pk[:-1] - pk[1:]), 0)
        return pk, torch.cat([torch.zeros_like(z[:1]), z])

    def heating(self, dp, nf):
        pk = self.levels(dp) ** ic.KAPPA
        play = (pk[1:] - pk[:-1]) / torch.log(pk[1:] / pk[:-1])
        return (nf[1:] - nf[:-1]) / (ic.CP_DRY * dp / self.st.gravity) / play

    def cgrid(self, dp, pt, ud, vd, dt, nf):
        dtdx, dtdy, ra, L = dt * self.rdx, dt * self.rdy, self.ra, self.L
        uc = 0.5 * (0.5 * (ud + _at(ud, -1, 0)) + 0.5 * (_at(ud, 0, 1) + _at(ud, -1, 1)))
        vc = 0.5 * (0.5 * (vd + _at(vd, 0, -1)) + 0.5 * (_at(vd, 1, 0) + _at(vd, 1, -1)))
        dpc, ptc = self.mass(dp, pt, uc, vc, dt, 'unconstrained', None if nf is None else self.heating(dp, nf))
        pk, gz = self.column(dpc, ptc)
        # A-grid winds of the top layer, used for every layer
        ut, vt = ud[L - 1:], vd[L - 1:]
        ua = 0.5 * (uc[L - 1:] + 0.25 * (_at(ut, 1, 0) + ut + _at(ut, 1, 1) + _at(ut, 0, 1)))
        va = 0.5 * (vc[L - 1:] + 0.25 * (_at(vt, 0, 1) + vt + _at(vt, 1, 1) + _at(vt, 1, 0)))
        ke = 0.5 * (va * _flux(_at(vc, 0, 1), dtdy * va, 0, 1, 'unconstrained')
                    + ua * _flux(_at(uc, 1, 0), dtdx * ua, 1, 0, 'unconstrained'))
        vor = self.st.coriolis - (uc - _at(uc, 0, -1)) * self.rdy + (vc - _at(vc, -1, 0)) * self.rdx
        um, vm = _at(ud, -1, 0), _at(vd, 0, -1)
        tu = _inner(vor, dtdx * um, dtdx * ud, 1 / (1 - dtdx * (ud - um)), 1, 0, ra)
        tv = _inner(vor, dtdx * vm, dtdx * vd, 1 / (1 - dtdy * (vd - vm)), 0, 1, ra)
        lap = self.lap(vor)

        def force(i, j):
            p0, p1, z0, z1 = pk[:-1], pk[1:], gz[:-1], gz[1:]
            q0, q1, y0, y1 = _at(p0, -i, -j), _at(p1, -i, -j), _at(z0, -i, -j), _at(z1, -i, -j)
            return ((p0 - q1) * (y0 - z1) + (q0 - p1) * (y1 - z0)) / (p0 - q1 + q0 - p1)
        fy = _flux(_at(tu, 0, 1), dtdx * vd, 0, 1, 'unconstrained')
        fx = _flux(_at(tv, 1, 0), dtdx * ud, 1, 0, 'unconstrained')
        u = uc + dt * (vd * fy + self.vy * (_at(lap, 0, 1) - lap)) - dtdx * (ke - _at(ke, -1, 0) - force(1, 0))
        v = vc - dt * (ud * fx + self.vx * (_at(lap, 1, 0) - lap)) - dtdy * (ke - _at(ke, 0, -1) - force(0, 1))
        return dpc, ptc, u, v

    def corners(self, q):
        a, b = (-1 / 12, 7 / 12, 7 / 12, -1 / 12), (-1 / 32, 9 / 32, 9 / 32, -1 / 32)
        a, b = ([float(np.float32(v)) for v in w] for w in (a, b))
        along = lambda f, w, i, j: sum(w[n] * _at(f, (n - 2) * i, (n - 2) * j) for n in range(4))  # noqa: E731
        return along(along(q, a, 1, 0), b, 0, 1) + along(along(q, a, 0, 1), b, 1, 0)

    def dgrid(self, dp, pt, ud, vd, cgrid, dt, nf):
        dtdx, dtdy, ra, L = dt * self.rdx, dt * self.rdy, self.ra, self.L
        dpc, _, uc, vc = cgrid
        new_dp, new_pt = self.mass(dp, pt, uc, vc, dt, 'nonnegative', None if nf is None else self.heating(dpc, nf))
        pk, gz = self.column(new_dp, new_pt)
        pb, zb = self.corners(pk), self.corners(gz)
        pb = torch.cat([pb[:-1], pk[-1:]])
        ut, vt = uc[L - 1:], vc[L - 1:]
        ub, vb = 0.5 * (ut + _at(ut, 0, -1)), 0.5 * (vt + _at(vt, -1, 0))
        ke = 0.5 * (vb * _flux(vd, dtdy * vb, 0, 1, 'constrained') + ub * _flux(ud, dtdx * ub, 1, 0, 'constrained'))
        vor = self.st.coriolis - (_at(ud, 0, 1) - ud) * self.rdy + (_at(vd, 1, 0) - vd) * self.rdx
        dv = self.rdx * (ud - _at(ud, -1, 0)) + self.rdy * (vd - _at(vd, 0, -1))
        dv = self.div * self.lap(self.lap(dv))
        un, vn = _at(ut, 1, 0), _at(vt, 0, 1)
        tu = _inner(vor, dtdx * ut, dtdx * un, 1 / (1 - dtdx * (un - ut)), 1, 0, ra)
        tv = _inner(vor, dtdx * vt, dtdx * vn, 1 / (1 - dtdy * (vn - vt)), 0, 1, ra)
        lap = self.lap(vor)

        def force(i, j):
            p0, p1, z0, z1 = pb[:-1], pb[1:], zb[:-1], zb[1:]
            q0, q1, y0, y1 = _at(p0, i, j), _at(p1, i, j), _at(z0, i, j), _at(z1, i, j)
            return ((q0 - p1) * (z0 - y1) + (p0 - q1) * (z1 - y0)) / (q0 - p1 + p0 - q1)
        fy = _flux(tu, dtdx * vt, 0, 1, 'constrained')
        fx = _flux(tv, dtdx * ut, 1, 0, 'constrained')
        g = ke - dv
        u = ud + dt * (vc * fy + self.vy * (lap - _at(lap, 0, -1))) - dtdx * (_at(g, 1, 0) - g - force(1, 0))
        v = vd - dt * (uc * fx + self.vx * (lap - _at(lap, -1, 0))) - dtdy * (_at(g, 0, 1) - g - force(0, 1))
        return new_dp, new_pt, u, v

    # -- vertical remap
    def interface_values(self, var, c):
        """Limited edge values (bottom, top) and curvature of each layer."""
        L, gam, lv = self.L, [None] * (self.L + 1), [None] * (self.L + 1)
        al = (c[L - 1] - c[L - 2]) / (c[L] - c[L - 1])
        be = al * (0.5 + al)
        lv[L] = (2 * al * (1 + al) * var[L - 1] + var[L - 2]) / be
        gam[L - 1] = (1 + al * (1.5 + al)) / be
        for k in range(L - 1, 0, -1):
            al = (c[k + 1] - c[k]) / (c[k] - c[k - 1])
            be = 2 + 2 * al - gam[k]
            lv[k] = (3 * (var[k] + al * var[k - 1]) - lv[k + 1]) / be
            gam[k - 1] = al / be
        be = 1 + al * (1.5 + al)
        lv[0] = (2 * al * (1 + al) * var[0] + var[1] - be * lv[1]) / (al * (0.5 + al) - be * gam[0])
        for k in range(1, L + 1):
            lv[k] = lv[k] - gam[k - 1] * lv[k - 1]
        for k in (L - 1, 1):
            lv[k] = _max(_min(lv[k], _max(var[k], var[k - 1])), _min(var[k], var[k - 1]))
        for k in range(2, L):
            lo, hi = _min(var[k - 1], var[k]), _max(var[k - 1], var[k])
            low, high = _max(lv[k], lo), _min(lv[k], hi)
            if k == L - 1:
                lv[k] = _max(high, lo)
            else:
                g2, g0 = gam[k + 1], gam[k - 1]
                lv[k] = torch.where(g2 * g0 > 0, _max(high, lo), torch.where(g2 > 0, low, high))
        btm, top = [lv[k] for k in range(L)], [lv[k + 1] for k in range(L)]

        def clamp(x, a, b, d):
            return _min(_max(x, _min(_min(a, b), d)), _max(_max(a, b), d))
        for k in range(2, L):
            p = var[k] - 2 * gam[k - 1]
            top[k] = clamp(top[k], var[k], p, p + 1.5 * gam[k - 2])
            p = var[k] + 2 * gam[k]
            btm[k] = clamp(btm[k], var[k], p, p - 1.5 * gam[k - 1])
        return btm, top, [6 * var[k] - 3 * (top[k] + btm[k]) for k in range(L)]

    def remap_column(self, var, c, d):
        """Layer means of var on interfaces c over the layers between interfaces d."""
        btm, top, cv = self.interface_values(var, c)
        d0, d1 = d[:-1], d[1:]
        out, third = torch.zeros_like(d0), float(np.float32(2 / 3))
        for k in range(self.L):
            s0, s1 = c[k], c[k + 1]
            hit = (s1 < d0) & (s0 > d1)
            ds = s1 - s0
            a, b, f = (d0 - s0) / ds, (d1 - s0) / ds, ds / (d1 - d0)
            t3, am, ap, t1 = 2 * a * a, a - 1, a + 1, a + b
            low, high = (d1 <= s1) & (s1 < d0) & (d0 < s0), (s1 < d1) & (d1 < s0) & (s0 <= d0)
            whole, inside = (d1 <= s1) & (s0 <= d0), (s1 < d1) & (d0 < s0)
            zero = torch.zeros_like(out)
            part = torch.where(low, am / 6 * (3 * (btm[k] * am - top[k] * ap) + cv[k] * (t3 - ap)), zero)
            part = part + torch.where(high, b / 2 * (btm[k] * (2 - b) + b * (top[k] + cv[k] * (1 - third * b))), zero)
            part = part + torch.where(whole, var[k].expand_as(out), zero)
            part = part + torch.where(inside, (a - b) / 6 * (3 * (btm[k] * (t1 - 2) - top[k] * t1)
                                                             + cv[k] * (t3 + t1 * (2 * b - 3))), zero)
            out = out + torch.where(hit, part * f, zero)
        return out

    def remap(self, dp, pt, ud, vd, old_u, old_v):
        """The winds' ring outside the domain is that of the step before, as the
        time loop remaps before it fills the halo."""
        def ringed(new, old, n):
            f = torch.nn.functional.pad(old[None], (n, n, n, n), mode='circular')[0]
            f[:, n:-n, n:-n] = new
            return f
        lev = self.levels(dp)
        tgt = torch.cat([self.ak[:-1, None, None] + self.bk[:-1, None, None] * (lev[:1] - self.ptop),
                         torch.full_like(lev[:1], self.ptop)])
        wide = [torch.nn.functional.pad(t[None], (3, 3, 3, 3), mode='circular')[0] for t in (lev, tgt)]
        c7, c1 = float(np.float32(7 / 12)), float(np.float32(1 / 12))
        winds = []
        for new, old, i, j in ((ud, old_u, 0, 1), (vd, old_v, 1, 0)):
            def face(t):
                ny, nx = t.shape[-2] - 4, t.shape[-1] - 4
                cut = lambda n: t[:, 2 + n * j:2 + n * j + ny, 2 + n * i:2 + n * i + nx]  # noqa: E731
                return c7 * (cut(0) + cut(-1)) - c1 * (cut(1) + cut(-2))
            winds.append(self.remap_column(ringed(new, old, 1), face(wide[0]), face(wide[1])))

        def energy_winds(u, v):
            cu = lambda i, j: u[:, 1 + j:u.shape[1] - 1 + j, 1 + i:u.shape[2] - 1 + i]  # noqa: E731
            cv = lambda i, j: v[:, 1 + j:v.shape[1] - 1 + j, 1 + i:v.shape[2] - 1 + i]  # noqa: E731
            ua = 0.25 * (cu(0, 0) + cu(0, 1)) + 0.125 * (cu(-1, 0) + cu(-1, 1) + cu(1, 0) + cu(1, 1))
            va = 0.25 * (cv(0, 0) + cv(1, 0)) + 0.125 * (cv(0, -1) + cv(1, -1) + cv(0, 1) + cv(1, 1))
            return ua * ua + va * va
        pk, tpk = lev ** ic.KAPPA, tgt ** ic.KAPPA
        cv_dry = ic.CP_DRY - ic.R_DRY
        gz = torch.cat([torch.zeros_like(lev[:1]), torch.cumsum(ic.CP_DRY * pt * (pk[:-1] - pk[1:]), 0)])
        mean = (pk[1:] - pk[:-1]) / torch.log(pk[1:] / pk[:-1])
        en = cv_dry * pt * mean + 0.5 * (gz[1:] + gz[:-1] + energy_winds(ringed(ud, old_u, 1), ringed(vd, old_v, 1)))
        er = self.remap_column(en, lev, tgt)
        tmean = (tpk[1:] - tpk[:-1]) / torch.log(tpk[1:] / tpk[:-1])
        w2 = energy_winds(*winds)
        z, out = torch.zeros_like(lev[0]), []
        for k in range(self.L):
            dpk = tpk[k] - tpk[k + 1]
            t = (er[k] - z - 0.5 * w2[k]) / (cv_dry * tmean[k] + 0.5 * ic.CP_DRY * dpk)
            z = z + ic.CP_DRY * t * dpk
            out.append(t)
        inner = [w[:, 1:-1, 1:-1] for w in winds]
        return tgt[:-1] - tgt[1:], torch.stack(out), inner[0], inner[1]

    # -- column physics
    def tendencies(self, dp, pt, ud, vd, nf):
        lev = self.levels(dp)
        pk = lev ** ic.KAPPA
        play = (pk[1:] - pk[:-1]) / torch.log(lev[1:] / lev[:-1]) / ic.KAPPA
        ua = (0.25 * (ud + _at(ud, 0, 1)) + 0.125 * (_at(ud, -1, 0) + _at(ud, -1, 1) + _at(ud, 1, 0) + _at(ud, 1, 1)))
        va = (0.25 * (vd + _at(vd, 1, 0)) + 0.125 * (_at(vd, 0, -1) + _at(vd, 1, -1) + _at(vd, 0, 1) + _at(vd, 1, 1)))
        gz = torch.cat([torch.zeros_like(lev[:1]), torch.cumsum(ic.CP_DRY * pt * (pk[:-1] - pk[1:]), 0)])
        cv_dry = ic.CP_DRY - ic.R_DRY
        en = cv_dry * pt * play + 0.5 * (gz[1:] + gz[:-1] + ua * ua + va * va)
        u, v, e = list(ua), list(va), list(en)
        for k in range(self.L - 1):
            du, dv = ua[k + 1] - ua[k], va[k + 1] - va[k]
            ri = ((pt[k + 1] - pt[k]) * (dp[k] * (gz[k + 1] - gz[k]) + dp[k + 1] * (gz[k + 2] - gz[k + 1]))
                  / ((dp[k] * pt[k] + dp[k + 1] * pt[k + 1]) * (du * du + dv * dv + float(np.float32(1e-4)))))
            t = 1 - (ri / 0.25).clamp(min=0)
            mix = torch.where(ri < 0.25, t * t * dp[k] * dp[k + 1] / (dp[k] + dp[k + 1]), torch.zeros_like(ri))
            for w in (u, v, e):
                x = mix * (w[k] - w[k + 1])
                w[k], w[k + 1] = w[k] - x / dp[k], w[k + 1] + x / dp[k + 1]
        z, tend = torch.zeros_like(lev[0]), []
        for k in range(self.L):
            dpk = pk[k] - pk[k + 1]
            t = (e[k] - z - 0.5 * (u[k] ** 2 + v[k] ** 2)) / (cv_dry * play[k] + 0.5 * ic.CP_DRY * dpk)
            z = z + ic.CP_DRY * t * dpk
            tend.append((t - pt[k]) / 600.0)
        return (torch.stack(tend), (torch.stack(u) - ua) / 600.0, (torch.stack(v) - va) / 600.0,
                nf[0] / (41680.0 * 5))

    def radiation(self, go, dp, pt, ts):
        """Net flux on the interfaces, bottom to top."""
        L, dev = self.L, self.dev
        tab = {n: torch.tensor(getattr(go, n), device=dev) for n in
               ('pressures', 'temperatures', 'sw_absorption', 'sw_scattering', 'lw_absorption',
                'planck_temperatures', 'planck', 'irradiance_fraction')}
        lev = self.levels(dp)
        pk, plog = lev ** ic.KAPPA, torch.log(lev[:-1] / lev[1:])
        play = dp / plog
        tlay = pt * (pk[:-1] - pk[1:]) / (plog * ic.KAPPA)
        lp, ll = torch.log(play), torch.log(lev)
        lo = torch.tensor([0] + list(range(L - 1)) + [L - 2], device=dev)
        a, b = lp[lo], lp[lo + 1]
        tlev = (tlay[lo] * (b - ll) + tlay[lo + 1] * (ll - a)) / (b - a)
        dm = dp / self.st.gravity

        def weight(x, grid):
            k = torch.searchsorted(grid, x.contiguous()).clamp(1, grid.numel() - 1)
            return k, (x - grid[k - 1]) / (grid[k] - grid[k - 1])
        kp, wp = weight(play, tab['pressures'])
        grids = tab['temperatures']

        def row(kr):
            g = grids[kr]                                    # (..., n_t)
            kt = torch.searchsorted(g, tlay[..., None].contiguous()).clamp(1, g.shape[-1] - 1)
            lo_t, hi_t = g.gather(-1, kt - 1), g.gather(-1, kt)
            return kt[..., 0], ((tlay[..., None] - lo_t) / (hi_t - lo_t))[..., 0]
        rows = [(kp - 1, 1 - wp) + row(kp - 1), (kp, wp) + row(kp)]

        def lookup(t):
            return sum(w * (t[kr, kt - 1] * (1 - wt) + t[kr, kt] * wt) for kr, w, kt, wt in rows)
        kl, wl = weight(tlev, tab['planck_temperatures'])
        ks, ws = weight(ts, tab['planck_temperatures'])
        xc, yc = (torch.tensor(v, device=dev) for v in ic.cell_axes(self.st))
        r = torch.sqrt(xc[None, :] ** 2 + yc[:, None] ** 2) / float(np.float32(100000e3))
        sun = 600.0 * (1 + float(np.float32(0.2)) / (1 + r * r))
        pi, albedo = float(np.float32(math.pi)), float(np.float32(0.3))
        emis = float(np.float32(0.99))
        net = torch.zeros_like(lev)

        def adding(R, T, su, sd, alb, em, down):
            A, E, B = [alb], [em], []
            for k in range(L):
                be = 1 / (1 - R[k] * A[k])
                B.append(be)
                E.append(su[k] + T[k] * be * (E[k] + sd[k] * A[k]))
                A.append(R[k] + T[k] * T[k] * be * A[k])
            up, dn = [None] * (L + 1), [None] * (L + 1)
            dn[L], up[L] = down, A[L] * down + E[L]
            for k in range(L - 1, -1, -1):
                dn[k] = B[k] * (sd[k] + T[k] * dn[k + 1] + R[k] * E[k])
                up[k] = A[k] * dn[k] + E[k]
            return torch.stack(up), torch.stack(dn)
        for g in range(go.n_g):
            # shortwave: asymmetry 0, overhead sun; the rescaling leaves its parameters as they are
            ka, sca = lookup(tab['sw_absorption'][g]), tab['sw_scattering'][g]
            tau, ssa = (ka + sca) * dm, sca / (ka + sca)
            g1, g2, g3, g4 = (7 - 4 * ssa) / 4, (4 * ssa - 1) / 4, 0.5, 0.5
            a1, a2 = g1 * g4 + g2 * g3, g2 * g3 + g2 * g4
            lam = torch.sqrt(g1 * g1 - g2 * g2)
            em, direct = torch.exp(-lam * tau), torch.exp(-tau)
            e2 = em * em
            n1 = ssa / ((1 - lam * lam) * (lam + g1 + (lam - g1) * e2))
            refl = n1 * ((1 - lam) * (a2 + lam * g3) - (1 + lam) * (a2 - lam * g3) * e2
                         - 2 * lam * (g3 - a2) * em * direct)
            tran = n1 * (2 * lam * (g4 + a1) * em - direct * ((1 + lam) * (a1 + lam * g4)
                                                              - (1 - lam) * (a1 - lam * g4) * e2))
            beam = [None] * (L + 1)
            beam[L] = tab['irradiance_fraction'][g] * sun
            for k in range(L - 1, -1, -1):
                beam[k] = direct[k] * beam[k + 1]
            beam = torch.stack(beam)
            g1, g2 = 2 * (1 - ssa * 0.5), ssa
            lam = torch.sqrt(g1 * g1 - g2 * g2)
            n1 = 1 / (lam + g1 + (lam - g1) * e2)
            up, dn = adding(n1 * g2 * (1 - e2), 2 * n1 * lam * em, refl * beam[1:], tran * beam[1:],
                            torch.full_like(ts, albedo), torch.zeros_like(ts), beam[L])
            net = net + (dn + beam) - up
            # longwave: no scattering, Planck source linear in optical depth
            tau = lookup(tab['lw_absorption'][g]) * dm
            T = torch.exp(-2 * tau)
            plk = tab['planck'][g]
            b = plk[kl - 1] * (1 - wl) + plk[kl] * wl
            bs = plk[ks - 1] * (1 - ws) + plk[ks] * ws
            diff = (1 - T) * (b[:-1] - b[1:]) / (2 * tau)
            up, dn = adding(torch.zeros_like(T), T, pi * (b[1:] - T * b[:-1] + diff),
                            pi * (b[:-1] - T * b[1:] - diff), torch.full_like(ts, 1 - emis), emis * pi * bs,
                            torch.zeros_like(ts))
            net = net + dn - up
        return net

    def forecast(self, fields, dt, steps, remap_every, go=None, ts=None):
        dp, pt, ud, vd = fields
        nf = tend = None
        for n in range(1, steps + 1):
            if go is not None:
                if n == 1:
                    nf = self.radiation(go, dp, pt, ts)
                tend = self.tendencies(dp, pt, ud, vd, nf)
            old_u, old_v = ud, vd
            cg = self.cgrid(dp, pt, ud, vd, dt / 2, nf)
            dp, pt, ud, vd = self.dgrid(dp, pt, ud, vd, cg, dt, nf)
            if tend is not None:
                c7, c1 = float(np.float32(7 / 12)), float(np.float32(1 / 12))
                ut, vt = tend[1], tend[2]
                pt, ts = pt + dt * tend[0], ts + dt * tend[3]
                ud = ud + dt * (c7 * (ut + _at(ut, 0, -1)) - c1 * (_at(ut, 0, 1) + _at(ut, 0, -2)))
                vd = vd + dt * (c7 * (vt + _at(vt, -1, 0)) - c1 * (_at(vt, 1, 0) + _at(vt, -2, 0)))
            if n % remap_every == 0:
                dp, pt, ud, vd = self.remap(dp, pt, ud, vd, old_u, old_v)
        return dp, pt, ud, vd, ts


def exact(case, seed):
    kind = case['kind']
    cells = _sizes(case)[0]
    if kind == 'ensemble':
        out = []
        for i, (s, n, L) in enumerate(_members(case)):
            f = _fields(s, n, n, L, seed * 100 + i)[:4]
            st = _blank(case, s, n, n, L)
            with torch.no_grad():
                out.append(list(_Scheme(st, f[0].device).forecast(f, st.dt, case['steps'], case['remap_every'])[:4]))
        return out
    limit = EXACT_GRADIENT if kind == 'gradient' else EXACT_FORWARD
    if cells * case['steps'] > limit:
        return None
    st = _blank(case, case['state'], case['nx'], case['ny'], case['nlay'])
    f = _fields(case['state'], case['nx'], case['ny'], case['nlay'], seed)
    sch = _Scheme(st, f[0].device)
    if kind == 'gradient':
        x = [t.detach().requires_grad_() for t in f[:4]]
        out = sch.forecast(x, st.dt, case['steps'], case['remap_every'])
        th2 = out[1] * out[1]
        loss = (th2 * gaussian_mask(st, case['radius'], th2.device) if case['radius'] else th2).sum()
        loss.backward()
        return {'loss': loss.detach(), 'gradients': [t.grad for t in x]}
    with torch.no_grad():
        if kind == 'physics':
            out = sch.forecast(f[:4], st.dt, case['steps'], case['remap_every'], gas_optics.synthetic(1), f[4])
            return {'fields': list(out[:4]), 'stable': 1, 'surface': [out[4]]}
        out = sch.forecast(f[:4], st.dt, case['steps'], case['remap_every'])
    return {'fields': list(out[:4]), 'stable': 1, 'surface': []}
