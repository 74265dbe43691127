"""The workloads that the library's speed is judged on.

Each case is one call pattern of a user of ``coseis_b200``, over the sizes of
the shipped configurations (bench.py, tests/sordcases.py):

  coupled   a program that advances a small model one step at a time through
            a ``Solver`` handle and reads the whole state back after each:
            latency and launches count
  run       ``sord.run`` of a point-source explosion, from parameters to
            output files: the drop-in use
  steps     a ``Solver`` handle advanced some steps at a time, with receivers
            and velocity planes written as the run goes: flat, terrain and
            perturbed meshes, both arithmetics, PML on the sides and the
            bottom, free surface on top; with ``stress`` the stress tensor is
            written too, every step
  rupture   the same on a planar slip-weakening fault, fault planes written
  ensemble  ``sord.run_ensemble`` over rupture scenarios of uneven sizes
  adjoint   receiver traces and their gradients through
            ``adjoint.ReceiverTraces``: every state kept, or binomial
            checkpointing; free or PML faces

``exact`` restates the wave solver in 64 bits with plain torch operations.
"""
import math
import os
import shutil
import tempfile

import numpy as np
import torch

from coseis_b200 import _lib, adjoint, sord

AXES = 'xyz'
RHO, VP, VS = 2670.0, 6000.0, 3464.0
MOMENT = ('mxx', 'myy', 'mzz', 'myz', 'mzx', 'mxy')
STRESS = ('wxx', 'wyy', 'wzz', 'wyz', 'wzx', 'wxy')
FAULT = ('sum', 'svm', 'tsm', 'trup')
NT = 10 ** 6  # steps that a handle may take: far more than are asked of it


# ---------------------------------------------------------------- the cases
def _steps(name, mesh, shape, npml, steps, arithmetic, stress=False):
    nx, ny, nz = shape
    c = {'kind': 'steps', 'mesh': mesh, 'nx': nx, 'ny': ny, 'nz': nz, 'npml': npml, 'steps': steps,
         'arithmetic': arithmetic, 'stress': stress}
    return dict(c, name=name) if name else c


def listed():
    return [
        # a coupling program's smallest call: one step, the state read back
        {'name': 'coupled_24', 'kind': 'coupled', 'nx': 24, 'ny': 24, 'nz': 24, 'npml': 4, 'arithmetic': 'reference'},
        # the shipped explosion configuration, whole, in the default arithmetic
        {'name': 'run_explosion_61', 'kind': 'run', 'nx': 61, 'ny': 61, 'nz': 61, 'npml': 10, 'steps': 200,
         'arithmetic': 'reference'},
        # a small production model on a flat mesh
        _steps('steps_flat_96', 'flat', (96, 80, 72), 10, 20, 'fast'),
        # terrain at an odd size, between the tests' and the benchmark's
        _steps('steps_terrain_odd', 'terrain', (203, 149, 97), 12, 20, 'fast'),
        # the benchmark's terrain model at 1/27 of its nodes, bit-exact arithmetic
        _steps('steps_terrain_256_ref', 'terrain', (256, 256, 128), 12, 10, 'reference'),
        # the same at 3/10 of its nodes, fast arithmetic: the largest
        _steps('steps_terrain_512', 'terrain', (512, 512, 256), 12, 20, 'fast'),
        # the reference's benchmark problem: a perturbed (general) mesh, random initial velocity
        _steps('steps_noise_160', 'noise', (160, 144, 120), 10, 20, 'fast'),
        # stress output at every step (each stage in its own kernel)
        _steps('steps_stress_96_ref', 'flat', (96, 80, 64), 8, 10, 'reference', stress=True),
        # the planar rupture configuration at half its linear size
        {'name': 'rupture_300', 'kind': 'rupture', 'nx': 300, 'ny': 150, 'nz': 150, 'npml': 10, 'steps': 20,
         'arithmetic': 'fast'},
        # a batch of rupture scenarios on one GPU
        {'name': 'ensemble_8', 'kind': 'ensemble', 'count': 8, 'least': 64, 'most': 128, 'npml': 10, 'steps': 100,
         'arithmetic': 'fast'},
        # gradients with every state kept, free faces
        {'name': 'adjoint_64', 'kind': 'adjoint', 'nx': 64, 'ny': 64, 'nz': 64, 'npml': 0, 'steps': 120,
         'snapshots': 0},
        # gradients with PML and binomial checkpointing
        {'name': 'adjoint_pml_56', 'kind': 'adjoint', 'nx': 60, 'ny': 56, 'nz': 52, 'npml': 8, 'steps': 80,
         'snapshots': 10},
    ]


def _between(rng, lo, hi):
    """A whole number in [lo, hi], even over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['coupled', 'run', 'steps', 'steps', 'steps', 'steps', 'rupture', 'ensemble', 'adjoint'])
    both = rng.choice(['reference', 'fast'])
    if kind == 'coupled':
        return {'kind': kind, 'nx': _between(rng, 20, 40), 'ny': _between(rng, 20, 40), 'nz': _between(rng, 20, 40),
                'npml': rng.randint(3, 6), 'arithmetic': both}
    if kind == 'run':
        return {'kind': kind, 'nx': _between(rng, 40, 80), 'ny': _between(rng, 40, 80), 'nz': _between(rng, 40, 80),
                'npml': rng.randint(5, 12), 'steps': rng.randint(80, 200), 'arithmetic': both}
    if kind == 'steps':
        mesh = rng.choice(['flat', 'terrain', 'noise'])
        most = 512 if both == 'fast' and mesh != 'noise' else 256
        shape = (_between(rng, 64, most), _between(rng, 64, most), _between(rng, 48, most // 2))
        return _steps(None, mesh, shape, rng.randint(6, 12), rng.randint(8, 20), both,
                      max(shape) <= 160 and rng.random() < 0.2)
    if kind == 'rupture':
        return {'kind': kind, 'nx': _between(rng, 80, 300), 'ny': _between(rng, 64, 150), 'nz': _between(rng, 64, 150),
                'npml': 10, 'steps': rng.randint(10, 20), 'arithmetic': both}
    if kind == 'ensemble':
        return {'kind': kind, 'count': rng.randint(4, 12), 'least': 64, 'most': 16 * rng.randint(5, 8), 'npml': 10,
                'steps': rng.randint(40, 100), 'arithmetic': both}
    return {'kind': kind, 'nx': _between(rng, 36, 64), 'ny': _between(rng, 36, 64), 'nz': _between(rng, 36, 64),
            'npml': rng.choice([0, 6, 8]), 'steps': rng.randint(40, 100), 'snapshots': rng.choice([0, 0, 8, 12])}


# ------------------------------------------------------------------- inputs
def _rng(seed, stream):
    return np.random.default_rng([int(seed), stream])


def _device():
    return 'cuda' if torch.cuda.is_available() else 'cpu'


def _normal(shape, seed, stream):
    g = torch.Generator(device=_device()).manual_seed(int(seed) * 64 + stream)
    return torch.randn(shape, generator=g, device=_device())


def _smooth(a):
    """A few passes of a three-point mean along each axis."""
    for d in range(a.dim()):
        for _ in range(4):
            a = (a + torch.roll(a, 1, d) + torch.roll(a, -1, d)) / 3.0
    return a / a.std()


def _shape(case):
    return case['nx'], case['ny'], case['nz']


def _spacing(case):
    return (50.0, 0.004) if case.get('mesh') == 'terrain' else (100.0, 0.008)


def _fields(case, seed):
    """Material (cells) and coordinates (nodes) as float32 arrays [l, k, j];
    names that are absent keep the mesh and medium of the parameters."""
    nx, ny, nz = _shape(case)
    dx, _ = _spacing(case)
    out = {}
    if case['mesh'] == 'terrain':
        x = torch.arange(nx, device=_device()) * dx
        y = torch.arange(ny, device=_device()) * dx
        r = _rng(seed, 1)
        xc, yc = (nx - 1) * dx * r.uniform(0.4, 0.6), (ny - 1) * dx * r.uniform(0.4, 0.6)
        wide = 5000.0 * min(nx, ny) / 768.0
        peak = min(500.0, 0.1 * dx * nz)
        hill = peak * torch.exp(-((x[None] - xc) ** 2 + (y[:, None] - yc) ** 2) / (2 * wide * wide))
        down = torch.arange(nz, device=_device())[:, None, None]
        out['z'] = (dx * down - hill[None] * (1.0 - down / (nz - 1.0))).float()
        depth = dx * (torch.arange(nz - 1, device=_device()) + 0.5)
        vs = torch.where(depth < 1000.0, 1000.0, torch.where(depth < 4000.0, 2500.0, 3500.0))[:, None, None]
        rho = torch.where(depth < 1000.0, 2200.0, torch.where(depth < 4000.0, 2500.0, 2700.0))[:, None, None]
        dv = 0.05 * _smooth(_normal((nz - 1, ny - 1, nx - 1), seed, 2)).clamp(-3, 3)
        out['vs'] = (vs * (1 + dv)).float()
        out['vp'] = (math.sqrt(3.0) * vs * (1 + dv)).float()
        out['rho'] = (rho * (1 + dv)).float()
    if case['mesh'] == 'noise':
        n = (nz, ny, nx)
        inside = torch.zeros(n, device=_device())
        p = case['npml']
        inside[1:nz - p - 1, p + 1:ny - p - 1, p + 1:nx - p - 1] = 0.17 * dx
        for d in range(3):
            at = [1, 1, 1]
            at[2 - d] = -1
            i = (dx * torch.arange(n[2 - d], device=_device())).view(at)
            out[AXES[d]] = (i + inside * _normal(n, seed, 3 + d).clamp(-1.5, 1.5) / 1.5).float()
    return {k: a.contiguous().cpu().numpy() for k, a in out.items()}


def _velocity(case, seed):
    """Random initial velocity, [l, k, j] per component."""
    nx, ny, nz = _shape(case)
    return [_normal((nz, ny, nx), seed, 8 + i).cpu().numpy() for i in range(3)]


def _source(case, seed):
    """Position (cell-registered node index) and moment of a point source."""
    r = _rng(seed, 12)
    x = [math.floor(n * f * 64.0) / 64.0 for n, f in zip(_shape(case), r.uniform(0.4, 0.6, 3))]
    m = r.standard_normal(6)
    return x, [float(v) for v in m * (2e12 / math.sqrt((m * m).sum()))]


def _receivers(case, seed, count=8):
    """Surface receivers at fractional positions inside the PML."""
    r = _rng(seed, 13)
    lo = case['npml'] + 1.5
    at = lambda n: math.floor(r.uniform(lo, n - 1 - lo) * 64.0) / 64.0
    return [[at(case['nx']), at(case['ny']), 0.0] for _ in range(count)]


def _faces(case):
    """PML everywhere but on top, or free faces without PML."""
    if case['npml'] == 0:
        return {'bc1': ['free'] * 3, 'bc2': ['free'] * 3, 'npml': 0}
    return {'bc1': ['pml', 'pml', 'free'], 'bc2': ['pml'] * 3, 'npml': case['npml']}


def _basic(case, nt):
    dx, dt = _spacing(case)
    return {'shape': [case['nx'], case['ny'], case['nz'], nt], 'delta': [dx, dx, dx, dt], 'rho': [RHO], 'vp': [VP],
            'vs': [VS], 'gam': [0.1], 'hourglass': [1.0, 1.0], 'itstats': 10, **_faces(case)}


def _stage(prm, path):
    here = os.getcwd()
    os.chdir(path)
    try:
        sord.stage(prm)
    finally:
        os.chdir(here)
    with open(os.path.join(path, 'sord.in')) as fh:
        return fh.read()


class _Handle:
    """A solver in a directory of its own, and how far its files were read."""

    def __init__(self, prm, files, arithmetic):
        self.dir = tempfile.mkdtemp(prefix='sord_case_')
        for name, a in files.items():
            np.ascontiguousarray(a, dtype='<f4').tofile(os.path.join(self.dir, name + '.bin'))
        self.solver = _lib.Solver(self.dir, _stage(prm, self.dir))
        self.solver.set_arithmetic(arithmetic)
        self.seen = 0

    def record(self, name, count):
        """The floats that the last pass added to an output file."""
        return np.fromfile(os.path.join(self.dir, name), '<f4', count, offset=4 * count * self.seen)

    def __del__(self):
        if hasattr(self, 'solver'):
            self.solver.close()
        shutil.rmtree(self.dir, ignore_errors=True)


def _planes(case):
    """Output planes of a component: (name, slices, values)."""
    nx, ny, nz = _shape(case)
    last = [case['steps'] - 1, None, case['steps']]
    return [('top', [[], [], 0, last], nx * ny), ('mid', [[], ny // 2, [], last], nx * nz)]


def _steps_prm(case, seed, files):
    prm = _basic(case, NT)
    prm['itio'] = case['steps']
    for name in files:
        prm[name] = [([], '=<', name + '.bin')]
    x, moment = _source(case, seed)
    for f, m in zip(MOMENT, moment):
        prm[f] = [(x + [[]], '.', m, 'brune', 0.1)]
    for a in AXES:
        prm['v' + a] = [(at, '=>', '%s-v%s.bin' % (name, a)) for name, at, _ in _planes(case)]
        prm['v' + a] += [(r + [[]], '.>', 'r%d-v%s.bin' % (i, a)) for i, r in enumerate(_receivers(case, seed))]
    if case['stress']:
        for f in STRESS:
            prm[f] = [([[], case['ny'] // 2, [], []], '=>', f + '.bin')]
    return prm


def _run_prm(case, seed):
    prm = _basic(case, case['steps'])
    prm.update({'gam': [0.0], 'bc1': ['pml'] * 3, 'bc2': ['pml'] * 3, 'itio': 50})
    nx, ny, nz = _shape(case)
    c = [nx // 2, ny // 2, nz // 2]
    size = 1e16 * float(_rng(seed, 14).uniform(0.5, 2.0))
    for f in MOMENT[:3]:
        prm[f] = [(c + [[]], '.', size, 'brune', 0.1)]
    for a in AXES:
        prm['v' + a] = [([[], c[1], [], [0, None, 10]], '=>', 'snap-v%s.bin' % a)]
        prm['v' + a] += [(list(r) + [[]], '=>', 'rec%d-v%s.bin' % (i, a)) for i, r in enumerate(_points(case, seed))]
    return prm


def _points(case, seed, count=8):
    r = _rng(seed, 15)
    p = case['npml'] + 2
    return [[int(r.integers(p, n - p)) for n in _shape(case)] for _ in range(count)]


def _stress_plane(shape, seed, stream, mean, std):
    """Seeded, smooth initial shear stress on a fault plane."""
    a = _smooth(torch.from_numpy(_rng(seed, stream).standard_normal(shape)))
    return (mean + std * a.numpy())


def _rupture_prm(case, seed, stream=20):
    """A slip-weakening fault on the z mid-plane, and its stress file."""
    nx, ny, nz = _shape(case)
    r = _rng(seed, stream)
    mus, mud, dc = (float(r.uniform(*b)) for b in ((0.6, 0.7), (0.45, 0.55), (0.2, 0.5)))
    tn = float(r.uniform(60e6, 120e6))
    ts = _stress_plane((ny, nx), seed, stream + 1, 0.58 * tn, 0.03 * tn)
    rj, rk = nx // 6, ny // 6
    half = max(1, min(15, (nx - 2 * rj) // 6, (ny - 2 * rk) // 6))
    ts[ny // 2 - half:ny // 2 + half, nx // 2 - half:nx // 2 + half] = 1.02 * mus * tn
    prm = {
        'shape': [nx, ny, nz, NT], 'delta': [100.0, 100.0, 100.0, 0.008], 'rho': [RHO], 'vp': [VP], 'vs': [VS],
        'gam': [0.1], 'hourglass': [1.0, 2.0], 'bc1': ['pml'] * 3, 'bc2': ['pml'] * 3, 'npml': case['npml'],
        'faultnormal': '+z', 'hypocenter': [nx // 2, ny // 2, nz * 0.5 - 0.5], 'vrup': -1.0,
        'mus': [1e4, ([[rj, nx - rj], [rk, ny - rk]], '=', mus)], 'mud': [mud], 'dc': [dc], 'tn': [-tn],
        'ts': [([], '=<', 'ts.bin')], 'itstats': 10,
    }
    return prm, ts.astype('<f4')


def _scenarios(case, seed):
    """Rupture scenarios of uneven sizes, which the case alone sets:
    (parameters, stress file) each."""
    r = _rng(case['count'], 17)
    out = []
    for i in range(case['count']):
        n = [16 * int(r.integers(case['least'] // 16, m // 16 + 1)) for m in (case['most'], 96, 96)]
        one = {'nx': n[0], 'ny': min(n[1], case['most']), 'nz': min(n[2], case['most']), 'npml': case['npml']}
        prm, ts = _rupture_prm(one, seed, 100 + 2 * i)
        prm['shape'][3] = case['steps']
        prm['itio'] = case['steps']
        for f in FAULT:
            prm[f] = [([[], [], -1], '=>', f + '.bin')]
        out.append((prm, ts))
    return out


def _adjoint_inputs(case, seed):
    """rho, vp, vs [j, k, l], moment, receivers and the recorded traces."""
    nx, ny, nz = _shape(case)
    n = (nx - 1, ny - 1, nz - 1)
    a = [(v * (1 + 0.03 * _smooth(_normal(n, seed, 30 + i)).clamp(-3, 3))).float().cpu()
         for i, v in enumerate((2700.0, VP, VS))]
    x, m = _source(case, seed)
    lo = case['npml'] + 2
    r = _rng(seed, 35)
    rec = [[int(r.integers(lo, nx - lo)), int(r.integers(lo, ny - lo)), 0] for _ in range(8)]
    seen = 1e-3 * _smooth(torch.from_numpy(r.standard_normal((8, 3, case['steps'])))).float()
    return a + [torch.tensor(m, dtype=torch.float64)], x, rec, seen


def _adjoint_prm(case):
    prm = _basic(case, case['steps'])
    for f in ('rho', 'vp', 'vs'):
        del prm[f]
    prm.update({'gam': [0.05], 'vpml': 4000.0, 'itio': 100})
    return prm


def prepare(case, seed):
    kind = case['kind']
    if kind == 'coupled':
        s = _Handle(_basic(case, NT), {}, case['arithmetic'])
        for a, v in zip(AXES, _velocity(case, seed)):
            s.solver.set_field('v' + a, v.T)
        s.solver.step(1)
        return {'case': case, 'handle': s}
    if kind == 'steps':
        files = _fields(case, seed)
        s = _Handle(_steps_prm(case, seed, files), files, case['arithmetic'])
        for a, v in zip(AXES, _velocity(case, seed)):
            s.solver.set_field('v' + a, v.T)
        return {'case': case, 'handle': s}
    if kind == 'rupture':
        prm, ts = _rupture_prm(case, seed)
        prm['itio'] = case['steps']
        last = [case['steps'] - 1, None, case['steps']]
        for f in FAULT:
            prm[f] = [([[], [], last], '=>', f + '.bin')]
        return {'case': case, 'handle': _Handle(prm, {'ts': ts}, case['arithmetic'])}
    if kind == 'run':
        return {'case': case, 'prm': _run_prm(case, seed)}
    if kind == 'ensemble':
        return {'case': case, 'scenarios': _scenarios(case, seed)}
    v, x, rec, seen = _adjoint_inputs(case, seed)
    problem = adjoint.Problem(_adjoint_prm(case), {'x': x, 'pulse': 'brune', 'tau': 0.1}, rec,
                              snapshots=case['snapshots'])
    return {'case': case, 'v': v, 'problem': problem, 'seen': seen}


# --------------------------------------------------------------------- runs
def run(state):
    case = state['case']
    return globals()['_run_' + case['kind']](case, state)


def _run_coupled(case, state):
    s = state['handle'].solver
    s.step(1)
    return {f + a: s.field(f + a) for f in 'vu' for a in AXES}


def _run_steps(case, state):
    h = state['handle']
    h.solver.step(case['steps'])
    nx, ny, nz = _shape(case)
    out = {}
    for a in AXES:
        for name, _, n in _planes(case):
            out['%s-v%s' % (name, a)] = h.record('%s-v%s.bin' % (name, a), n)
        out['traces-v' + a] = np.stack([h.record('r%d-v%s.bin' % (i, a), case['steps']) for i in range(8)])
    if case['stress']:
        for f in STRESS:
            out[f] = h.record(f + '.bin', (nx - 1) * (nz - 1) * case['steps'])
    h.seen += 1
    return out


def _run_rupture(case, state):
    h = state['handle']
    h.solver.step(case['steps'])
    out = {f: h.record(f + '.bin', case['nx'] * case['ny']) for f in FAULT}
    h.seen += 1
    return out


def _run_run(case, state):
    os.environ['SORD_ARITHMETIC'] = case['arithmetic']
    here, d = os.getcwd(), tempfile.mkdtemp(prefix='sord_case_')
    try:
        os.chdir(d)
        sord.run(state['prm'])
        # components together: one may vanish by symmetry
        return {'snap': np.stack([np.fromfile('snap-v%s.bin' % a, '<f4') for a in AXES]),
                'rec': np.stack([[np.fromfile('rec%d-v%s.bin' % (i, a), '<f4') for i in range(8)] for a in AXES])}
    finally:
        os.chdir(here)
        shutil.rmtree(d, ignore_errors=True)
        del os.environ['SORD_ARITHMETIC']


def _run_ensemble(case, state):
    os.environ['SORD_ARITHMETIC'] = case['arithmetic']
    d = tempfile.mkdtemp(prefix='sord_case_')
    try:
        dirs = [os.path.join(d, 's%03d' % i) for i in range(case['count'])]
        for at, (_, ts) in zip(dirs, state['scenarios']):
            os.makedirs(at)
            ts.tofile(os.path.join(at, 'ts.bin'))
        sord.run_ensemble([prm for prm, _ in state['scenarios']], dirs)
        return [np.stack([np.fromfile(os.path.join(at, f + '.bin'), '<f4') for f in FAULT]) for at in dirs]
    finally:
        shutil.rmtree(d, ignore_errors=True)
        del os.environ['SORD_ARITHMETIC']


def _run_adjoint(case, state):
    v = [a.clone().requires_grad_() for a in state['v']]
    traces = adjoint.ReceiverTraces.apply(*v, state['problem'])
    loss = 0.5 * ((traces - state['seen']) ** 2).sum()
    loss.backward()
    return {'traces': traces.detach(), 'rho': v[0].grad, 'vp': v[1].grad, 'vs': v[2].grad, 'moment': v[3].grad}


# --------------------------------------------------------------------- work
def _node_bytes(case):
    """Bytes of one node-update: v, u in and out, mr and gam, lam, mu, yy and
    1/V, the coordinates that vary, and per PML slab that the node and its
    cell lie in the memory of three components in and out."""
    mesh = case.get('mesh', 'flat')
    n = 48 + 8 + 16 + {'flat': 0, 'terrain': 4, 'noise': 12}[mesh]
    p = case['npml']
    sides = 6 if case['kind'] in ('run', 'rupture', 'ensemble') else 5
    share = sum(p * (2 if d < 2 or sides == 6 else 1) / m for d, m in enumerate(_shape(case)))
    return n + 48 * share


def work(case):
    if case['kind'] == 'ensemble':
        mid = 8 * (case['least'] // 16 + case['most'] // 16)
        one = dict(case, nx=mid, ny=min(mid, 80), nz=min(mid, 80))
        updates = case['count'] * case['steps'] * one['nx'] * one['ny'] * one['nz']
    else:
        one = case
        updates = case.get('steps', 1) * case['nx'] * case['ny'] * case['nz']
    flops, size = 546.0 * updates, float(_node_bytes(one)) * updates
    if case['kind'] == 'adjoint':  # the forward run and the transposed one
        flops, size = 3 * flops, 3 * size
    if case['kind'] == 'coupled':
        size += 24.0 * updates
    return {'bytes': size, 'flops': flops}


# ------------------------------------------------------------ in 64 bits
class _Wave64:
    """The solver's equations in 64 bits on arrays [l, k, j]: support-operator
    gradients (the exact integrals of trilinear hexahedra), Hooke's law,
    stiffness and viscous hourglass control, split-field PML, leapfrog."""

    def __init__(self, prm, rho, vp, vs, x, device):
        f = lambda v: float(np.float32(v))
        self.n = prm['shape'][2::-1]
        self.dx = [f(v) for v in prm['delta'][:3]]
        self.dt = f(prm['delta'][3])
        self.hg = [f(v) for v in prm['hourglass']]
        self.gam = self.dt * f(prm['gam'][0])
        self.device = device
        self.brackets(x)
        mu = rho * vs * vs
        lam = rho * vp * vp - 2.0 * mu
        yy = mu * (lam + mu) / (lam + 2.0 * mu) * math.sqrt(sum(d * d for d in self.dx) / 3.0) / 12.0
        mass = self.zeros()
        for n in range(8):
            self.at(mass, n).add_(0.125 * rho * self.vol)
        self.lam, self.mu, self.yy, self.mr = lam, mu, yy, 1.0 / mass
        self.pml(prm, vp, vs)
        self.u, self.v, self.a = ([self.zeros() for _ in range(3)] for _ in range(3))
        self.g = [[0.0] * 3 for _ in range(3)]
        self.p = [[0.0] * 3 for _ in range(3)]

    def zeros(self):
        return torch.zeros(self.n, dtype=torch.float64, device=self.device)

    def at(self, a, n):
        """Node array at corner n = dj + 2 dk + 4 dl of every cell."""
        c = [(n >> (2 - i)) & 1 for i in range(3)]
        return a[c[0]:self.n[0] - 1 + c[0], c[1]:self.n[1] - 1 + c[1], c[2]:self.n[2] - 1 + c[2]]

    def brackets(self, x):
        """B[d][n]: cell integral of dN_n/dx_d; the box formula, or exact
        2 x 2 x 2 Gauss quadrature of the trilinear map."""
        sign = [[(n >> d & 1) * 2 - 1 for n in range(8)] for d in range(3)]
        if x is None:
            vol = self.dx[0] * self.dx[1] * self.dx[2]
            self.B = [[sign[d][n] * 0.25 * vol / self.dx[d] for n in range(8)] for d in range(3)]
            self.vol = vol
            return
        self.B = [[0.0] * 8 for _ in range(3)]
        self.vol = 0.0
        at = [[self.at(a, n) for n in range(8)] for a in x]
        r = 1.0 / math.sqrt(3.0)
        for q in range(8):
            xi = [r * sign[d][q] for d in range(3)]
            dN = [[0.125 * sign[d][n] * math.prod(1 + sign[e][n] * xi[e] for e in range(3) if e != d)
                   for n in range(8)] for d in range(3)]
            J = [[sum(dN[d][n] * at[c][n] for n in range(8)) for d in range(3)] for c in range(3)]
            # cofactors: d(x_d)/d(xi_e) of the inverse times the determinant
            C = [[J[(c + 1) % 3][(d + 1) % 3] * J[(c + 2) % 3][(d + 2) % 3] -
                  J[(c + 1) % 3][(d + 2) % 3] * J[(c + 2) % 3][(d + 1) % 3] for d in range(3)] for c in range(3)]
            self.vol = self.vol + sum(J[0][d] * C[0][d] for d in range(3))
            for c in range(3):
                for n in range(8):
                    self.B[c][n] = self.B[c][n] + sum(dN[d][n] * C[c][d] for d in range(3))

    def pml(self, prm, vp, vs):
        n = prm['npml']
        t = lambda a, d: torch.tensor(a, dtype=torch.float64, device=self.device).view([-1 if i == 2 - d else 1 for i in range(3)])
        self.cell, self.node, self.inner, self.any = [], [], True, False
        if n == 0:
            return
        vpml = prm.get('vpml', -1.0)
        if vpml <= 0:
            lo, hi = float(torch.as_tensor(vs).min()), float(torch.as_tensor(vp).max())
            vpml = 2.0 * lo * hi / (lo + hi)
        damp = 3.5 * vpml / math.sqrt(sum(d * d for d in self.dx) / 3.0) * (8 / 15 + (-3 / 100 + n / 1500) * n) / n ** 2
        dn = lambda i: damp * i * i
        dc = lambda i: damp * (i * i + (i - 1) ** 2) * 0.5
        dt = self.dt
        for d in range(3):
            m = prm['shape'][d]
            ends = [prm['bc1'][d] == 'pml', prm['bc2'][d] == 'pml']
            node = [max(n - i if ends[0] else 0, n - (m - 1 - i) if ends[1] else 0, 0) for i in range(m)]
            cell = [max(n - i if ends[0] else 0, n - (m - 2 - i) if ends[1] else 0, 0) for i in range(m - 1)]
            self.node.append([t([i > 0 for i in node], d) > 0, t([-2 * dn(i) / (2 + dt * dn(i)) for i in node], d),
                              t([2 / (2 + dt * dn(i)) for i in node], d)])
            self.cell.append([t([i > 0 for i in cell], d) > 0, t([(2 - dt * dc(i)) / (2 + dt * dc(i)) for i in cell], d),
                              t([2 * dt / (2 + dt * dc(i)) for i in cell], d)])
            self.inner = self.inner & ~self.node[d][0]
            self.any = self.any | self.cell[d][0]

    def grad(self, f, d):
        return sum(self.at(f, n) * self.B[d][n] for n in range(8))

    def spread(self, terms):
        """Node sums of terms(n), the cell values for corner n."""
        f = self.zeros()
        for n in range(8):
            self.at(f, n).add_(terms(n))
        return f

    def step(self, source=()):
        """One step; source: (component, cell slices, stress added)."""
        dt, g = self.dt, self.gam
        self.v = [v + dt * a for v, a in zip(self.v, self.a)]
        self.u = [u + dt * v for u, v in zip(self.u, self.v)]
        G = [[None] * 3 for _ in range(3)]
        for i in range(3):
            for d in range(3):
                du, dv = self.grad(self.u[i], d), self.grad(self.v[i], d)
                s = du + g * dv
                if self.cell:
                    on, c1, c2 = self.cell[d]
                    mem = c2 * dv + c1 * self.g[d][i]
                    s = torch.where(on, mem, torch.where(self.any, du, s))
                    self.g[d][i] = torch.where(on, mem, 0.0)
                G[i][d] = s
        tr = self.lam * (G[0][0] + G[1][1] + G[2][2])
        S = {}
        for c, (i, j) in enumerate(((0, 0), (1, 1), (2, 2), (1, 2), (2, 0), (0, 1))):
            s = 2.0 * self.mu * G[i][i] + tr if i == j else self.mu * (G[i][j] + G[j][i])
            for comp, at, value in source:
                if comp == c:
                    if not s.requires_grad:
                        s = s.clone()
                    add = torch.zeros_like(s)
                    add[at] = value
                    s = s + add
            S[i, j] = S[j, i] = s / self.vol
        self.stress = [S[0, 0], S[1, 1], S[2, 2], S[1, 2], S[2, 0], S[0, 1]]
        f = []
        for i in range(3):
            total = 0.0
            for d in range(3):
                s = -self.spread(lambda n: S[i, d] * self.B[d][n])
                if self.node:
                    on, c1, c2 = self.node[d]
                    mem = c2 * s + c1 * self.p[d][i]
                    self.p[d][i] = torch.where(on, self.p[d][i] + dt * mem, 0.0)
                    s = torch.where(on, mem, s)
                total = total + s
            f.append(total - self.hourglass(i))
        self.a = [self.mr * s for s in f]

    def hourglass(self, i):
        k, h2 = self.hg[0], self.dt * self.hg[1]
        sign = [[(n >> d & 1) * 2 - 1 for n in range(8)] for d in range(3)]
        pattern = [[sign[1][n] * sign[2][n] for n in range(8)], [sign[0][n] * sign[2][n] for n in range(8)],
                   [sign[0][n] * sign[1][n] for n in range(8)],
                   [sign[0][n] * sign[1][n] * sign[2][n] for n in range(8)]]

        def force(w):
            m = [self.yy * sum(self.at(w, n) * p[n] for n in range(8)) for p in pattern]
            return self.spread(lambda n: sum(c * p[n] for c, p in zip(m, pattern)))
        f = force(k * self.u[i] + h2 * self.v[i])
        if self.node:
            f = torch.where(self.inner, f, force(h2 * self.v[i]) if h2 > 0 else 0.0)
        return f


def _brune(t, tau):
    return math.exp(-t / tau) * t / tau ** 2 if t > 0 else 0.0


def _weights(x, offset, shape):
    """Trilinear weights of a position: ((l, k, j), weight) per point."""
    x = [float(np.float32(v)) - offset for v in x]
    lo = [math.floor(v) for v in x]
    out = []
    for c in np.ndindex(2, 2, 2):
        i = [a + b for a, b in zip(lo, c)]
        w = math.prod(1.0 - abs(v - a) for v, a in zip(x, i))
        if all(0 <= a < n for a, n in zip(i, shape)) and w:
            out.append((tuple(i[::-1]), w))
    return out


def _d(v, device):
    return torch.as_tensor(np.ascontiguousarray(v), dtype=torch.float64, device=device)


def exact(case, seed):
    kind = case['kind']
    if kind in ('rupture', 'ensemble'):
        # friction and rupture times switch on thresholds: a 64-bit run may
        # take the other branch a step earlier or later
        return None
    device = _device()
    if kind == 'adjoint':
        # every step's tensors are kept: about 300 fields a step
        if case['nx'] * case['ny'] * case['nz'] * case['steps'] > 4e7:
            return None
        return _exact_adjoint(case, seed, device)
    with torch.no_grad():
        return globals()['_exact_' + kind](case, seed, device)


def _whole(case, device):
    n = (case['nz'] - 1, case['ny'] - 1, case['nx'] - 1)
    return [torch.full(n, v, dtype=torch.float64, device=device) for v in (RHO, VP, VS)]


def _exact_coupled(case, seed, device):
    m = _Wave64(_basic(case, 1), *_whole(case, device), None, device)
    m.v = [_d(v, device) for v in _velocity(case, seed)]
    m.step()
    m.step()
    return {f + a: getattr(m, f)[i].cpu().numpy().T for f in 'vu' for i, a in enumerate(AXES)}


def _exact_steps(case, seed, device):
    files = _fields(case, seed)
    prm = _steps_prm(case, seed, files)
    nx, ny, nz = _shape(case)
    mat = _whole(case, device)
    for i, f in enumerate(('rho', 'vp', 'vs')):
        if f in files:
            mat[i] = _d(files[f], device)
    x = None
    if case['mesh'] != 'flat':
        dx = _spacing(case)[0]
        x = [_d(files[a], device) if a in files else
             (dx * torch.arange(n, dtype=torch.float64, device=device)).view([-1 if i == 2 - d else 1 for i in range(3)])
             .expand(nz, ny, nx) for d, (a, n) in enumerate(zip(AXES, (nx, ny, nz)))]
    m = _Wave64(dict(prm, rho=None), *mat, x, device)
    m.v = [_d(v, device) for v in _velocity(case, seed)]
    at, moment = _source(case, seed)
    where = _weights(at, 0.5, (nx - 1, ny - 1, nz - 1))
    probes = [_weights(r, 0.0, (nx, ny, nz)) for r in _receivers(case, seed)]
    traces = [[[] for _ in probes] for _ in AXES]
    planes = {f: [] for f in STRESS}
    for it in range(case['steps']):
        tf = _brune(it * m.dt, 0.1)
        m.step([(c, q, float(np.float32(v)) * tf * w) for c, v in enumerate(moment) for q, w in where])
        for i in range(3):
            for r, pr in enumerate(probes):
                traces[i][r].append(sum(w * m.v[i][q] for q, w in pr))
        if case['stress']:
            for f, s in zip(STRESS, m.stress):
                planes[f].append(s[:, ny // 2, :].reshape(-1).clone())
    out = {}
    for i, a in enumerate(AXES):
        out['top-v' + a] = m.v[i][0].reshape(-1).cpu().numpy()
        out['mid-v' + a] = m.v[i][:, ny // 2, :].reshape(-1).cpu().numpy()
        out['traces-v' + a] = np.array([[float(s) for s in t] for t in traces[i]])
    if case['stress']:
        for f in STRESS:
            out[f] = torch.cat(planes[f]).cpu().numpy()
    return out


def _exact_run(case, seed, device):
    prm = _run_prm(case, seed)
    nx, ny, nz = _shape(case)
    m = _Wave64(prm, *_whole(case, device), None, device)
    c = [nx // 2, ny // 2, nz // 2]
    size = float(np.float32(prm['mxx'][0][2]))
    where = _weights(c, 0.5, (nx - 1, ny - 1, nz - 1))
    rec = _points(case, seed)
    snap, seen = [], []
    for it in range(case['steps']):
        tf = _brune(it * m.dt, 0.1)
        m.step([(i, q, size * tf * w) for i in range(3) for q, w in where])
        if it % 10 == 0:
            snap.append(torch.stack([v[:, c[1], :].reshape(-1) for v in m.v]))
        seen.append(torch.stack([torch.stack([v[l, k, j] for j, k, l in rec]) for v in m.v]))
    return {'snap': torch.cat(snap, -1).cpu().numpy(), 'rec': torch.stack(seen, -1).cpu().numpy()}


def _exact_adjoint(case, seed, device):
    (rho, vp, vs, moment), x, rec, seen = _adjoint_inputs(case, seed)
    nx, ny, nz = _shape(case)
    v = [a.to(device, torch.float64).requires_grad_() for a in (rho, vp, vs, moment.float())]
    m = _Wave64(_adjoint_prm(case), *[a.permute(2, 1, 0) for a in v[:3]], None, device)
    where = _weights(x, 0.5, (nx - 1, ny - 1, nz - 1))
    traces = []
    for it in range(case['steps']):
        tf = _brune(it * m.dt, 0.1)
        m.step([(c, q, v[3][c] * (tf * w)) for c in range(6) for q, w in where] if tf else ())
        traces.append(torch.stack([torch.stack([m.v[i][l, k, j] for i in range(3)]) for j, k, l in rec]))
    traces = torch.stack(traces, -1)
    loss = 0.5 * ((traces - seen.to(device, torch.float64)) ** 2).sum()
    loss.backward()
    return {'traces': traces.detach().cpu(), **{f: a.grad.cpu() for f, a in zip(('rho', 'vp', 'vs', 'moment'), v)}}
