"""Workloads by which the framework's speed is measured.

Every case is one call sequence of a user's program through the public entry
points, at sizes of the tests, of the benchmark and of sample-scale runs:

  engine  one report interval of a running engine, as permeability.converge
          makes it: the steps, the error check, the flux and convergence sums,
          and the dense fields; with `checkpoint` the dense populations too.  Single phase (2-D and 3-D, body force or
          pressure inlet and outlet) and two phases, each storage type.
  batch   one report interval of many uneven media in one launch.
  conv    one layer of the warm-start operator in training: forward, data,
          weight and bias gradients.
  net     one inference of the learned mobility network with its shipped
          weights.
  darcy   the block pressure solve of the in-run correction.

listed() holds the fixed cases, draw() gives others of the same ranges,
prepare() makes what a program has in hand, run() is one pass, work() what a
pass cannot do without and exact() the pass's result in FP64 by plain torch.
"""
import math
from pathlib import Path

import numpy as np
import torch

import lbflow_b200
from lbflow_b200 import Engine, batch, conv, warmstart

FORCE = 1e-5                # body force of the permeability runs, along x
COLOR_FORCE = 2e-6          # of the two-phase runs, along z
SIGMA, BETA, ANGLE = 1e-3, 0.7, 60.0
COLOR_TAU = (1.0, 0.7)
SLOPE = 0.1                 # leaky ReLU of the operator
WEIGHTS = Path(lbflow_b200.__file__).resolve().parent / 'weights' / 'mobility.pt'


def listed():
    return [
        # A validation run: small 2-D medium, launches and latency only.
        _engine('plane-48x40', 48, 40, 0, steps=400, collision='SRT', tau=0.9, porosity=0.5, sigma=2.0),
        # A small crop of a scan, the size of the precision tests.
        _engine('crop-48', 48, 48, 48, steps=400),
        # Odd extents, pressure inlet and outlet planes, and a checkpoint.
        _engine('pressure-161x93x117', 161, 93, 117, steps=100, collision='SRT', porosity=0.3, boundary='pressure',
                checkpoint=True),
        # The benchmark's cube: the reference's FP64 arithmetic throughout.
        _engine('cube-256-fp64', 256, 256, 256, steps=100, sigma=3.0),
        # The same with reduced storage, for time to permeability.
        _engine('cube-256-fp32', 256, 256, 256, steps=100, sigma=3.0, storage='fp32'),
        _engine('cube-192-fp16', 192, 192, 192, steps=100, sigma=3.0, storage='fp16'),
        # Two-phase displacement: a crop at reduced storage, and the benchmark's medium.
        _engine('color-48x48x96-fp32', 48, 48, 96, steps=100, model='color', storage='fp32', porosity=0.3, sigma=2.0,
                checkpoint=True),
        _engine('color-128x128x256', 128, 128, 256, steps=40, model='color', porosity=0.3, sigma=2.0),
        # Many media in one launch.
        dict(name='batch-48', kind='batch', count=48, low=32, high=96, steps=200, storage='fp64'),
        # The operator's heaviest layer in a training step.
        dict(name='conv-train-64', kind='conv', op='conv3', cin=64, cout=64, batch=2, nx=48, ny=48, nz=48),
        # The mobility network on a whole medium.
        dict(name='net-96', kind='net', nx=96, ny=96, nz=96, porosity=0.22, sigma=3.0),
        # The correction of a 192^3 run on 2^3 blocks.
        dict(name='darcy-96', kind='darcy', nx=96, ny=96, nz=96),
    ]


def _engine(name, nx, ny, nz, steps, model='scsp', collision='MRT', storage='fp64', tau=1.0, porosity=0.22,
            sigma=3.0, boundary='force', checkpoint=False):
    return dict(name=name, kind='engine', model=model, collision=collision, storage=storage, nx=nx, ny=ny, nz=nz,
                steps=steps, tau=tau, porosity=porosity, sigma=sigma, boundary=boundary, checkpoint=checkpoint)


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['plane', 'medium', 'medium', 'pressure', 'color', 'color', 'batch', 'conv', 'net', 'darcy'])
    if kind == 'plane':
        return _unnamed(_engine('', _log_uniform(rng, 30, 400), _log_uniform(rng, 30, 400), 0, rng.randint(100, 400),
                                collision=rng.choice(['SRT', 'MRT']), tau=round(rng.uniform(0.7, 1.3), 2),
                                porosity=round(rng.uniform(0.4, 0.6), 2), sigma=round(rng.uniform(2.0, 4.0), 1)))
    if kind in ('medium', 'pressure'):
        edge = [_log_uniform(rng, 32, 250) for _ in range(3)]
        pressure = kind == 'pressure'
        return _unnamed(_engine('', *edge, rng.randint(30, 100),
                                collision='SRT' if pressure else rng.choice(['SRT', 'MRT']),
                                storage='fp64' if pressure else rng.choice(['fp64', 'fp64', 'fp32', 'fp16']),
                                tau=round(rng.uniform(0.8, 1.2), 2), porosity=round(rng.uniform(0.18, 0.35), 2),
                                sigma=round(rng.uniform(2.0, 5.0), 1), boundary='pressure' if pressure else 'force',
                                checkpoint=rng.random() < 0.25))
    if kind == 'color':
        return _unnamed(_engine('', *[_log_uniform(rng, 32, 150) for _ in range(3)], rng.randint(10, 40),
                                model='color', storage=rng.choice(['fp64', 'fp64', 'fp32']),
                                porosity=round(rng.uniform(0.25, 0.35), 2), sigma=round(rng.uniform(2.0, 3.0), 1),
                                checkpoint=rng.random() < 0.25))
    if kind == 'batch':
        return dict(kind='batch', count=rng.randint(4, 48), low=32, high=rng.choice([48, 64, 96]),
                    steps=rng.randint(64, 200), storage=rng.choice(['fp64', 'fp32', 'fp16']))
    if kind == 'conv':
        op = rng.choice(['conv3', 'conv3', 'down2', 'up2'])
        cin, cout = rng.choice([(16, 16), (32, 32), (64, 64), (128, 64), (128, 128)] if op == 'conv3' else
                               [(16, 32), (32, 64), (64, 128)])
        if op == 'up2':
            cin, cout = cout, cin
        edge = [2 * _log_uniform(rng, 6, 24) for _ in range(3)]
        return dict(kind='conv', op=op, cin=cin, cout=cout, batch=rng.randint(1, 2), nx=edge[0], ny=edge[1], nz=edge[2])
    if kind == 'net':
        edge = [8 * _log_uniform(rng, 4, 12) for _ in range(3)]
        return dict(kind='net', nx=edge[0], ny=edge[1], nz=edge[2], porosity=round(rng.uniform(0.18, 0.35), 2),
                    sigma=round(rng.uniform(2.0, 5.0), 1))
    edge = [rng.choice([16, 24, 32, 40, 48, 64, 80, 96]) for _ in range(3)]
    while _coarsest(edge) > 1024:
        edge = [rng.choice([16, 24, 32, 40, 48, 64, 80, 96]) for _ in range(3)]
    return dict(kind='darcy', nx=edge[0], ny=edge[1], nz=edge[2])


def _unnamed(case):
    del case['name']
    return case


def _coarsest(edge):
    """Cells of the coarsest grid the block solve halves `edge` down to."""
    edge = list(edge)
    while math.prod(edge) > 512 and not any(n % 2 for n in edge):
        edge = [n // 2 for n in edge]
    return math.prod(edge)


# ------------------------------------------------------------------ inputs --
def _generator(seed):
    return torch.Generator(device='cuda').manual_seed(int(seed))


def _smooth_noise(shape, sigma, gen):
    """White noise through a periodic Gaussian filter of width sigma."""
    f = torch.fft.rfftn(torch.randn(shape, generator=gen, device='cuda'))
    for ax, n in enumerate(shape):
        k = torch.fft.rfftfreq(n, device='cuda') if ax == len(shape) - 1 else torch.fft.fftfreq(n, device='cuda')
        view = [1] * len(shape)
        view[ax] = -1
        f *= torch.exp(-2.0 * (math.pi * sigma * k) ** 2).reshape(view)
    return torch.fft.irfftn(f, s=shape)


def _medium(shape, sigma, porosity, gen):
    """Porous medium: the noise below its `porosity` quantile is pore space."""
    n = _smooth_noise(shape, sigma, gen)
    return n < n.flatten().kthvalue(max(1, int(porosity * n.numel()))).values


def _shape(case):
    return (case['nz'], case['ny'], case['nx']) if case['nz'] else (case['ny'], case['nx'])


def _engine_input(case, seed):
    """Label array (on the GPU) and label table of an engine case."""
    shape = _shape(case)
    fluid = _medium(shape, case['sigma'], case['porosity'], _generator(seed))
    g = torch.where(fluid, 75, 255).to(torch.uint8)
    if case['model'] == 'color':
        # The inlet third is filled with the displacing phase.
        g[:shape[0] // 3][fluid[:shape[0] // 3]] = 76
        return g, {75: ('GV', COLOR_FORCE, 5, 1), 76: ('GV', COLOR_FORCE, 5, 0), 255: ('SD', ANGLE, 0, 0)}
    if case['boundary'] == 'pressure':
        # Open planes at both x ends inside solid side walls.
        g[:, 0], g[:, -1], g[0], g[-1] = 255, 255, 255, 255
        g[1:-1, 1:-1, :2] = 75
        g[1:-1, 1:-1, -2:] = 75
        g[1:-1, 1:-1, 0] = 10
        g[1:-1, 1:-1, -1] = 11
        return g, {75: ('VD', 0.0, 0, 0), 10: ('PB', 1.0005, 1, 0), 11: ('PB', 0.9995, 2, 0), 255: ('SD', 90.0, 0, 0)}
    return g, {75: ('GV', FORCE, 1, 0), 255: ('SD', 90.0, 0, 0)}


def _batch_input(case, seed):
    """Media of uneven shapes and their relaxation times."""
    rng = np.random.default_rng(seed)
    gen = _generator(seed)
    edges = [e for e in (32, 48, 64, 96) if case['low'] <= e <= case['high']]
    shapes = np.random.default_rng(case['count']).choice(edges, size=(case['count'], 3)).tolist()
    geoms, taus = [], []
    for shape in map(tuple, shapes):
        fluid = _medium(shape, float(rng.uniform(1.5, 6.0)), float(rng.uniform(0.10, 0.35)), gen)
        geoms.append(torch.where(fluid, 75, 255).to(torch.uint8))
        taus.append(float(rng.uniform(0.6, 1.4)))
    return geoms, taus


def _conv_input(case, seed):
    gen = _generator(seed)
    dims = (case['batch'], case['nz'], case['ny'], case['nx'])
    out = {'conv3': dims, 'down2': (dims[0],) + tuple(d // 2 for d in dims[1:]),
           'up2': (dims[0],) + tuple(2 * d for d in dims[1:])}[case['op']]
    cin, cout = case['cin'], case['cout']
    wshape = {'conv3': (cout, cin, 3, 3, 3), 'down2': (cout, cin, 2, 2, 2), 'up2': (cin, cout, 2, 2, 2)}[case['op']]
    fan = cin if case['op'] == 'up2' else cin * wshape[-1] ** 3
    x = torch.randn(*dims, cin, generator=gen, device='cuda').to(torch.bfloat16)
    w = torch.randn(wshape, generator=gen, device='cuda') * math.sqrt(2.0 / fan)
    b = 0.1 * torch.randn(cout, generator=gen, device='cuda')
    gy = torch.randn(*out, cout, generator=gen, device='cuda').to(torch.bfloat16)
    return x, w, b, gy


def _net_input(case, seed):
    fluid = _medium(_shape(case), case['sigma'], case['porosity'], _generator(seed))
    return warmstart.features(fluid.unsqueeze(0))


def _darcy_input(case, seed):
    """Block mobilities with the contrast of a porous medium: log-normal, with
    a floor where a block holds no pores."""
    gen = _generator(seed)
    n = _smooth_noise(_shape(case), 1.5, gen).double()
    return torch.exp(2.0 * n / n.std()).clamp(min=1e-2)


# -------------------------------------------------------------------- runs --
def prepare(case, seed):
    if case['kind'] == 'engine':
        g, labels = _engine_input(case, seed)
        tau = COLOR_TAU if case['model'] == 'color' else (case['tau'],)
        eng = Engine(g.cpu().numpy(), labels, model=case['model'], collision=case['collision'], tau=tau,
                     rho=(1.0, 1.0), alpha0=1 / 3, sigma=SIGMA, beta=BETA, storage=case['storage'])
        eng.initialize()
        eng.convergence(first=True)
        per = 1 + (case['model'] == 'color') + eng.dims
        out = torch.empty(per * eng.N, dtype=torch.float64, device='cuda')
        rst = torch.empty(eng.phases * eng.q * eng.N if case['checkpoint'] else 0, dtype=torch.float64, device='cuda')
        return dict(kind='engine', engine=eng, steps=case['steps'], out=out, checkpoint=rst)
    if case['kind'] == 'batch':
        geoms, taus = _batch_input(case, seed)
        b = batch.Batch([g.cpu().numpy() for g in geoms], taus, {75: ('GV', FORCE, 1, 0), 255: ('SD', 90.0, 0, 0)},
                        storage=case['storage'])
        b.initialize()
        b.convergence(first=True)
        return dict(kind='batch', batch=b, steps=case['steps'])
    if case['kind'] == 'conv':
        x, w, b, gy = _conv_input(case, seed)
        return dict(kind='conv', op=case['op'], x=x.requires_grad_(), w=w.requires_grad_(), b=b.requires_grad_(), gy=gy)
    if case['kind'] == 'net':
        return dict(kind='net', net=warmstart.load_mobility(WEIGHTS)[0], x=_net_input(case, seed))
    return dict(kind='darcy', mob=_darcy_input(case, seed))


def run(state):
    if state['kind'] == 'engine':
        eng, out = state['engine'], state['out']
        eng.step(state['steps'] - 1, adjacent=True)
        eng.step(1, macros=True)
        eng.check()
        flux = eng.flux_sums()
        conv_sums = eng.convergence()
        eng.fields_dense_async(out.data_ptr(), out.numel())
        rst = state['checkpoint']
        if rst.numel():
            eng.populations_dense_async(rst.data_ptr(), rst.numel())
        eng.synchronize()
        scalars = out.numel() - eng.dims * eng.N
        got = dict(flux=flux, convergence=conv_sums, density=out[:scalars], velocity=out[scalars:])
        return dict(got, populations=rst) if rst.numel() else got
    if state['kind'] == 'batch':
        b = state['batch']
        b.step(state['steps'] - 1, adjacent=True)
        b.step(1, macros=True)
        b.check()
        conv_sums = b.convergence()
        flux = b.flux_sums()
        rho, u = b.macros(0)
        return dict(flux=flux, convergence=conv_sums, density=rho, velocity=u)
    if state['kind'] == 'conv':
        y = getattr(conv, state['op'])(state['x'], state['w'], state['b'], SLOPE)
        return (y.detach(),) + torch.autograd.grad(y, (state['x'], state['w'], state['b']), state['gy'])
    if state['kind'] == 'net':
        with torch.no_grad():
            return state['net'](state['x'])
    phi, iterations = warmstart.darcy_pressure_device(state['mob'], FORCE, 2)
    return dict(phi=phi, iterations=iterations)


# -------------------------------------------------------------------- work --
ELEM = {'fp64': 8, 'fp32': 4, 'fp16': 2}


def work(case):
    """Bytes and operations of one pass.  A time step reads and writes every
    population of every pore voxel once."""
    if case['kind'] == 'engine':
        q, phases = (19 if case['nz'] else 9), (2 if case['model'] == 'color' else 1)
        voxels = math.prod(_shape(case))
        nodes = case['porosity'] * voxels
        fields = 8 * voxels * (phases + (3 if case['nz'] else 2) + (phases * q if case['checkpoint'] else 0))
        # About 20 operations per population and phase in the collision.
        return dict(bytes=case['steps'] * nodes * 2 * phases * q * ELEM[case['storage']] + fields,
                    flops=case['steps'] * nodes * 20 * phases * q)
    if case['kind'] == 'batch':
        edges = [e for e in (32, 48, 64, 96) if case['low'] <= e <= case['high']]
        nodes = case['count'] * 0.225 * (sum(edges) / len(edges)) ** 3
        return dict(bytes=case['steps'] * nodes * 2 * 19 * ELEM[case['storage']], flops=case['steps'] * nodes * 20 * 19)
    if case['kind'] == 'conv':
        rows = case['batch'] * case['nx'] * case['ny'] * case['nz']
        taps = 27 if case['op'] == 'conv3' else 8
        if case['op'] == 'down2':
            rows //= 8
        out_rows = rows * 8 if case['op'] == 'up2' else rows
        in_rows = rows * 8 if case['op'] == 'down2' else rows
        # Forward, data gradient and weight gradient; input and its gradient,
        # output and its gradient, weights and theirs.
        return dict(flops=3 * 2 * rows * taps * case['cin'] * case['cout'],
                    bytes=4 * (in_rows * case['cin'] + out_rows * case['cout']) + 8 * taps * case['cin'] * case['cout'])
    voxels = case['nx'] * case['ny'] * case['nz']
    if case['kind'] == 'net':
        return dict(flops=warmstart.MobilityNet().flops(voxels), bytes=2 * 2 * 8 * voxels)
    # Per iteration the operator and one smoothing cycle; some thirty iterations.
    return dict(bytes=16 * voxels, flops=30 * 150 * voxels)


# ------------------------------------------------------------ FP64 results --
_E2 = [(0, 0), (1, 0), (0, 1), (-1, 0), (0, -1), (1, 1), (-1, 1), (-1, -1), (1, -1)]
_E3 = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (-1, 1, 0),
       (1, -1, 0), (-1, -1, 0), (1, 0, 1), (-1, 0, 1), (1, 0, -1), (-1, 0, -1), (0, 1, 1), (0, -1, 1), (0, 1, -1),
       (0, -1, -1)]


class _Lattice:
    """D2Q9 / D3Q19 on a dense periodic grid of voxels, x the last axis;
    populations are tensors (Q, grid), vectors (D, grid) in x, y, z order."""

    def __init__(self, fluid):
        self.D = fluid.dim()
        self.E = _E2 if self.D == 2 else _E3
        self.op = [self.E.index(tuple(-c for c in e)) for e in self.E]
        weight = {0: 4 / 9, 1: 1 / 9, 2: 1 / 36} if self.D == 2 else {0: 1 / 3, 1: 1 / 18, 2: 1 / 36}
        self.order = [sum(c != 0 for c in e) for e in self.E]
        self.e = torch.tensor(self.E, dtype=torch.float64, device=fluid.device)
        self.w = self.per_direction([weight[k] for k in self.order])
        self.fluid = fluid
        self.open = torch.stack([self.shift(fluid, e) for e in self.E])     # the voxel x - e_q is fluid

    def per_direction(self, values):
        return torch.tensor(values, dtype=torch.float64, device='cuda').reshape(-1, *[1] * self.D)

    def shift(self, v, e):
        """v at x - e."""
        return torch.roll(v, e, dims=[v.dim() - 1 - a for a in range(self.D)])

    def pull(self, f):
        moved = torch.stack([self.shift(f[q], e) for q, e in enumerate(self.E)])
        return torch.where(self.open, moved, f[self.op])

    def dot(self, v):
        """e_q . v for every direction."""
        return torch.tensordot(self.e, v, dims=1)

    def momentum(self, f):
        return torch.tensordot(self.e.T, f, dims=1)

    def equilibrium(self, rho, u):
        """The velocity part of the equilibrium, over the weights."""
        eu = self.dot(u)
        return rho * (3.0 * eu + 4.5 * eu * eu - 1.5 * (u * u).sum(0))

    def collide(self, f, feq, u, force, sp, sm):
        """Two-rate collision: even parts relax at sp, odd ones at sm, with
        the half-step body-force source."""
        eu, ef = self.dot(u), self.dot(force)
        src = self.w * (3.0 * (ef - (u * force).sum(0)) + 9.0 * eu * ef)
        d = f - feq
        even = -0.5 * sp * (d + d[self.op]) + 0.5 * (1 - 0.5 * sp) * (src + src[self.op])
        odd = -0.5 * sm * (d - d[self.op]) + 0.5 * (1 - 0.5 * sm) * (src - src[self.op])
        return (f + even + odd) * self.fluid


def _odd_rate(collision, sp):
    return 8.0 * (2.0 - sp) / (8.0 - sp) if collision == 'MRT' else sp


def _sums(lat, rho, u, u0, ua, phi=None, phi0=None, phia=None):
    """The report sums of the fields: flux and convergence."""
    m = lat.fluid
    zero = torch.zeros((), dtype=torch.float64, device=m.device)
    u3 = [u[a] if a < lat.D else torch.zeros_like(u[0]) for a in range(3)]
    share = m.double() if phi is None else rho[0] / (rho[0] + rho[1]).clamp(min=1e-300)
    flux = [x.sum() for x in u3] + [(share * x).sum() for x in u3]
    flux += [(rho[0] * m).sum(), (rho[1] * m).sum() if phi is not None else zero, (share * m).sum()]
    change = [((u - u0) ** 2).sum(), (u ** 2).sum(), ((u - ua) ** 2).sum()]
    change += [((phi - p) * m).abs().max() if phi is not None else zero for p in (phi0, phia)] + [zero]
    return torch.stack(flux).cpu().numpy(), torch.stack(change).cpu().numpy()


def _single_phase(g, force, collision, tau, steps, pressure=False):
    lat = _Lattice(g != 255)
    m, E = lat.fluid.double(), lat.E
    F = torch.stack([force * m if a == 0 else 0.0 * m for a in range(lat.D)])
    sp = 1.0 / tau
    sm = _odd_rate(collision, sp)

    def step(f, ends):
        rho, u = f.sum(0), (lat.momentum(f) + 0.5 * F) * m
        for label, density, s in ends:
            # The axial velocity that the known populations leave at the
            # prescribed density, and the unknown ones rebuilt.
            at = g == label
            known = sum((2.0 if e[0] else 1.0) * f[q] for q, e in enumerate(E) if e[0] != s)
            ux = -s * (known / density - 1.0)
            new = f.clone()
            for q, e in enumerate(E):
                if e[0] == s:
                    t = sum(n[d] * e[d] * f[k] for k, n in enumerate(E) if n[0] == 0 for d in (1, 2))
                    new[q] = torch.where(at, f[lat.op[q]] + 6.0 * s * lat.w[q] * density * ux - 0.5 * t, f[q])
            f = new
            rho = torch.where(at, density, rho)
            u = torch.stack([torch.where(at, ux if a == 0 else 0.0 * ux, u[a]) for a in range(lat.D)])
        return lat.collide(f, lat.w * (rho + lat.equilibrium(1.0, u)), u, F, sp, sm), rho * m, u

    # At t = 0 everything, the boundary planes too, is at rest.
    f, rho, u0 = step(lat.w * m - 1.5 * lat.w * lat.dot(F), [])
    u, ends = u0, [(10, 1.0005, 1), (11, 0.9995, -1)] if pressure else []
    for _ in range(steps):
        ua = u
        f, rho, u = step(lat.pull(f), ends)
    if pressure:
        # The boundary planes keep the reported velocity as their history.
        ua = torch.where((g == 10) | (g == 11), u, ua)
    return _sums(lat, [rho], u, u0, ua) + (rho, u, f)


def _two_phase(g, steps):
    """Color-gradient MRT with wall angle ANGLE (LBFlow's ColorFluid::Run)."""
    lat = _Lattice(g != 255)
    m, E = lat.fluid.double(), lat.E
    F = torch.stack([COLOR_FORCE * m if a == 2 else 0.0 * m for a in range(3)])
    a0 = 1 / 3
    rest = lat.per_direction([a0 if k == 0 else (1 - a0) / (12 * k) for k in lat.order])
    length = lat.per_direction([math.sqrt(max(k, 1)) for k in lat.order])
    pert = lat.per_direction([-1 / 3 if k == 0 else 1 / (18 * k) for k in lat.order])
    first = (g == 76).double()
    near = [lat.shift(lat.fluid, tuple(-c for c in e)) for e in E]     # x + e_q is fluid
    wall = lat.fluid & ~torch.stack(near).all(0)
    # Wall normal (toward the fluid) in the order z, y, x, and the rotation
    # that turns it onto the last axis.
    n = [-sum(e[2 - d] * (~near[q]).double() for q, e in enumerate(E)) for d in range(3)]

    def turn(o, a):
        h = torch.sqrt(o * o + a * a)
        safe = torch.where(h != 0, h, 1.0)
        return torch.where(h != 0, a / safe, 1.0), torch.where(h != 0, o / safe, 0.0)

    c1, s1 = turn(n[0], n[1])
    c2, s2 = turn(torch.sqrt(n[0] * n[0] + n[1] * n[1]), n[2])
    T = [[c1, -s1, 0 * c1], [c2 * s1, c2 * c1, -s2], [s2 * s1, s2 * c1, c2]]
    ca, sa = math.cos(ANGLE / 180 * math.pi), math.sin(ANGLE / 180 * math.pi)
    weight = lat.w.flatten().tolist()
    # Directions with a component along z, y, x, the positive ones first.
    along = [[q for s in (1, -1) for q, e in enumerate(E) if e[2 - d] == s] for d in range(3)]

    def gradient(phi):
        at = [lat.shift(phi, tuple(-c for c in e)) for e in E]
        gr = []
        for d in range(3):
            s = torch.zeros_like(phi)
            for q in along[d]:
                c = weight[q] * torch.where(wall, torch.where(near[q], at[q] - phi, 0.0), at[q])
                s = s + c if E[q][2 - d] == 1 else s - c
            gr.append(3.0 * s)
        norm = torch.sqrt(gr[0] * gr[0] + gr[1] * gr[1] + gr[2] * gr[2])
        gn = [T[r][0] * gr[0] + T[r][1] * gr[1] + T[r][2] * gr[2] for r in range(3)]
        c, s = turn(-gn[0], gn[1])
        # The contact angle in the rotated frame, turned back.
        t = [-s * (norm * sa), c * (norm * sa), norm * ca]
        rot = [T[0][r] * t[0] + T[1][r] * t[1] + T[2][r] * t[2] for r in range(3)]
        return [torch.where(wall, rot[d], gr[d]) for d in range(3)], norm

    def step(f0, f1):
        d0, d1 = f0.sum(0), f1.sum(0)
        dt = d0 + d1
        safe = torch.where(lat.fluid, dt, 1.0)
        phi = (d0 - d1) / safe
        tau = 0.5 * ((1 + phi) * COLOR_TAU[0] + (1 - phi) * COLOR_TAU[1])
        f = f0 + f1
        u = (lat.momentum(f) + 0.5 * F) / safe
        sp = 1.0 / tau
        f = lat.collide(f, rest * dt + lat.w * lat.equilibrium(dt, u), u, F, sp, _odd_rate('MRT', sp))
        gr, norm = gradient(phi)
        active = norm > 1e-9
        cosine = lat.dot(torch.stack(gr[::-1])) / torch.where(active, norm, 1.0)
        f = f + torch.where(active, 2.25 * SIGMA * norm / tau * (lat.w * cosine * cosine - pert), 0.0)
        side = BETA * d0 * d1 / safe ** 2 * cosine / length * (rest * dt)
        f0 = d0 / safe * f + torch.where(active, side, 0.0)
        return f0 * m, (f - f0) * m, d0 * m, d1 * m, u * m, phi

    start = rest * m - 1.5 * lat.w * lat.dot(F)
    f0, f1, d0, d1, u0, phi0 = step(start * first, start * (m - first))
    u, phi = u0, phi0
    for _ in range(steps):
        ua, phia = u, phi
        f0, f1, d0, d1, u, phi = step(lat.pull(f0), lat.pull(f1))
    return _sums(lat, [d0, d1], u, u0, ua, phi, phi0, phia) + (torch.cat([d0.flatten(), d1.flatten()]), u,
                                                                   torch.cat([f0, f1]))


def _conv_exact(x, w, op, adjoint=False):
    """The linear map of a layer on (B, D, H, W, C) in FP64."""
    w = w.double()
    if op == 'conv3':
        y = 0
        for k in range(27):
            d = (k // 9, k // 3 % 3, k % 3)
            y = y + torch.roll(x, [1 - v for v in d], dims=(1, 2, 3)) @ w[:, :, d[0], d[1], d[2]].T
        return y
    B, D, H, W, C = x.shape
    if op == 'down2':
        v = x.reshape(B, D // 2, 2, H // 2, 2, W // 2, 2, C).permute(0, 1, 3, 5, 2, 4, 6, 7)
        return v.reshape(B, D // 2, H // 2, W // 2, -1) @ w.permute(2, 3, 4, 1, 0).reshape(-1, w.shape[0])
    y = (x @ w.permute(0, 2, 3, 4, 1).reshape(C, -1)).reshape(B, D, H, W, 2, 2, 2, w.shape[1])
    return y.permute(0, 1, 4, 2, 5, 3, 6, 7).reshape(B, 2 * D, 2 * H, 2 * W, -1)


def _layer(x, w, b, op, slope=SLOPE):
    y = _conv_exact(x, w, op) + b.double()
    return torch.where(y > 0, y, slope * y) if slope is not None else y


def _net_exact(x):
    p = {k: v.cuda() for k, v in torch.load(WEIGHTS, map_location='cpu', weights_only=False)['state'].items()}

    def c3(name, v, skip=None, slope=SLOPE):
        v = v if skip is None else torch.cat([v, skip], dim=-1)
        return _layer(v, p[name + '_w'], p[name + '_b'], 'conv3', slope)

    def resize(name, v, op):
        return _layer(v, p[name + '_w'], p[name + '_b'], op)

    e1 = c3('enc1b', c3('enc1a', x))
    e2 = c3('enc2b', c3('enc2a', resize('down1', e1, 'down2')))
    e3 = c3('enc3b', c3('enc3a', resize('down2', e2, 'down2')))
    v = c3('midb', c3('mida', resize('down3', e3, 'down2')))
    v = c3('dec3b', c3('dec3a', resize('up3', v, 'up2'), e3))
    v = c3('dec2b', c3('dec2a', resize('up2', v, 'up2'), e2))
    v = c3('dec1b', c3('dec1a', resize('up1', v, 'up2'), e1))
    return c3('head', v, slope=None)


def _darcy_exact(mob, g, h):
    """Zero-mean pressure of the conserved block fluxes: conjugate gradients
    with the diagonal as preconditioner."""
    axes = (2, 1, 0)
    face = [torch.sqrt(mob * torch.roll(mob, -1, ax)) for ax in axes]

    def apply(p):
        out = torch.zeros_like(p)
        for f, ax in zip(face, axes):
            q = f * (torch.roll(p, -1, ax) - p)
            out -= q - torch.roll(q, 1, ax)
        return out / h ** 2

    diag = sum(f + torch.roll(f, 1, ax) for f, ax in zip(face, axes)) / h ** 2
    r = -g * (face[0] - torch.roll(face[0], 1, 2)) / h
    stop = 1e-12 * r.norm()
    p = torch.zeros_like(r)
    z = r / diag
    d = z.clone()
    rz = (r * z).sum()
    for it in range(20000):
        ad = apply(d)
        alpha = rz / (d * ad).sum()
        p += alpha * d
        r -= alpha * ad
        if it % 50 == 0 and r.norm() < stop:
            break
        z = r / diag
        rz, old = (r * z).sum(), rz
        d = z + rz / old * d
    return p - p.mean()


def exact(case, seed):
    if case['kind'] == 'engine':
        g, _ = _engine_input(case, seed)
        if case['model'] == 'color':
            flux, change, density, u, f = _two_phase(g, case['steps'])
        else:
            pressure = case['boundary'] == 'pressure'
            flux, change, density, u, f = _single_phase(g, 0.0 if pressure else FORCE, case['collision'], case['tau'],
                                                        case['steps'], pressure)
        got = dict(flux=flux, convergence=change, density=density.flatten(), velocity=u.movedim(0, -1).flatten())
        return dict(got, populations=f.flatten()) if case['checkpoint'] else got
    if case['kind'] == 'batch':
        # Every medium's sums; the fields of the first, as run() reads them.
        got = [_single_phase(g, FORCE, 'MRT', tau, case['steps']) for g, tau in zip(*_batch_input(case, seed))]
        return dict(flux=np.stack([v[0] for v in got]), convergence=np.stack([v[1] for v in got]),
                    density=got[0][2].cpu().numpy(), velocity=got[0][3].cpu().numpy())
    if case['kind'] == 'conv':
        x, w, b, gy = _conv_input(case, seed)
        x, w, b = (v.double().requires_grad_() for v in (x, w, b))
        y = _layer(x, w, b, case['op'])
        return (y.detach(),) + torch.autograd.grad(y, (x, w, b), gy.double())
    if case['kind'] == 'net':
        return _net_exact(_net_input(case, seed).double())
    return dict(phi=_darcy_exact(_darcy_input(case, seed), FORCE, 2.0), iterations=None)
