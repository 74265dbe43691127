"""The fast-arithmetic step kernel of rectilinear and terrain meshes
(csrc/modal.cuh) at the sizes and options where its tiles, planes and rules
change: one interior tile exactly, one node more, an interior one node wide,
a mesh that is PML almost throughout, sources in every class of box, each
hourglass setting, a sheared mesh (which takes the general kernels), and
moduli set between steps.  Against the FP64 oracle, held to the rule of
tests/test_fast_arithmetic.py: relative L2 error at most ten times the FP32
oracle's own, or 1e-6."""
import os

import numpy as np
import pytest

import sordcases as sc

NPML = 4


def flat(inner, nt=10, hourglass=(1.0, 2.0), gam=0.2, top='free'):
    """A mesh with `inner` interior nodes per axis (those whose cells lie
    outside the PML; a free top adds its PML-sized rows to the interior)."""
    n = [i + 2 * NPML + 2 for i in inner]
    prm = {
        'shape': n + [nt], 'delta': [100.0, 100.0, 100.0, 0.008],
        'rho': [2670.0], 'vp': [6000.0], 'vs': [3464.0], 'gam': [gam], 'hourglass': list(hourglass),
        'bc1': ['pml', 'pml', top], 'bc2': ['pml'] * 3, 'npml': NPML, 'itstats': 3, 'itio': 10,
    }
    # a source in the interior, in a slab of each axis, and in a corner
    at = [[n[0] / 2 + 0.3, n[1] / 2 - 0.2, n[2] / 2 + 0.1], [1.5, n[1] / 2, n[2] / 2], [n[0] / 2, n[1] - 2.5, n[2] / 2],
          [n[0] / 2, n[1] / 2, n[2] - 2.5], [1.5, 1.5, n[2] - 2.5]]
    prm['mxx'] = [(x + [[]], '.', 1e16 * (i + 1), 'brune', 0.05) for i, x in enumerate(at)]
    prm['myz'] = [(x + [[]], '.', -4e15, 'brune', 0.05) for x in at]
    prm['pxy'] = [(at[0] + [[]], '.', 1e5, 'brune', 0.05)]
    for f in ('vx', 'vy', 'vz', 'uz'):
        prm[f] = [([[], [], [], -1], '=>', 'vol-%s.bin' % f)]
    return prm


def terrain(inner, **kw):
    prm = flat(inner, **kw)
    prm['z'] = [([], '=<', 'z.bin')]
    return prm


def terrain_z(prm):
    nx, ny, nz = prm['shape'][:3]
    x, y, z = np.meshgrid(np.arange(nx), np.arange(ny), np.arange(nz), indexing='ij')
    top = 60.0 * np.sin(x / 3.0) * np.cos(y / 2.5)
    return (100.0 * z - top * (1.0 - z / (nz - 1.0))).astype('<f4')


def sheared(inner, **kw):
    """x = j + k / 2: rectilinear to the class test, but not boxes."""
    prm = flat(inner, **kw)
    prm['affine'] = [[1.0, 0.5, 0.0], [0.0, 1.0, 0.0], [0.0, 0.0, 1.0]]
    return prm


CASES = {
    'one_tile': lambda: flat((31, 7, 9)),
    'tile_and_one': lambda: flat((32, 8, 9)),
    'one_short': lambda: flat((30, 6, 5)),
    'one_wide': lambda: flat((1, 9, 8), top='pml'),
    'all_pml': lambda: flat((1, 1, 1), top='pml'),
    'no_viscous': lambda: flat((33, 9, 8), hourglass=(1.0, 0.0), gam=0.0),
    'no_stiffness': lambda: flat((33, 9, 8), hourglass=(0.0, 1.0)),
    'no_hourglass': lambda: flat((33, 9, 8), hourglass=(0.0, 0.0)),
    'sheared': lambda: sheared((33, 9, 8)),
    'terrain_one_tile': lambda: terrain((31, 7, 9)),
    'terrain_tile_and_one': lambda: terrain((32, 8, 9)),
    'terrain_one_wide': lambda: terrain((9, 1, 8)),
    'terrain_no_viscous': lambda: terrain((33, 9, 8), hourglass=(1.0, 0.0), gam=0.0),
}


def stage(prm, path, realsize=4):
    os.makedirs(path)
    if 'z' in prm:
        terrain_z(prm).astype('<f%d' % realsize).ravel(order='F').tofile(os.path.join(path, 'z.bin'))
    sc.stage(prm, path, realsize=realsize)


def read(path, size):
    """The output files by quantity, components together."""
    out = {}
    for f in sorted(os.listdir(path)):
        if f.startswith('vol-'):
            out.setdefault(f[4], []).append(np.fromfile(os.path.join(path, f), '<f%d' % size).astype(float))
    return {k: np.concatenate(v) for k, v in out.items()}


@pytest.mark.gpu
@pytest.mark.parametrize('name', sorted(CASES))
def test_modal_step_accuracy(name, tmp_path, oracle_bins, gpu_lib):
    prm = CASES[name]()
    o64, o32, fast = (str(tmp_path / d) for d in ('o64', 'o32', 'fast'))
    stage(prm, o64, 8)
    stage(prm, o32)
    stage(prm, fast)
    sc.run_oracle(o64, oracle_bins['f64'])
    sc.run_oracle(o32, oracle_bins['f32'])
    sc.run_gpu(fast, arithmetic='fast')
    a, b, c = read(fast, 4), read(o64, 8), read(o32, 4)
    assert sorted(a) == ['u', 'v']
    for k in a:
        n = np.linalg.norm(b[k])
        assert n > 0
        e, e32 = np.linalg.norm(a[k] - b[k]) / n, np.linalg.norm(c[k] - b[k]) / n
        assert e <= max(10 * e32, 1e-6), (k, e, e32)


@pytest.mark.gpu
def test_modal_step_moduli_set_between_steps(tmp_path, gpu_lib):
    """Moduli set between steps reach the next step: against a handle in
    reference order, ten steps, within 1e-5 of the field."""
    from coseis_b200 import _lib
    out = []
    for mode in ('reference', 'fast'):
        d = str(tmp_path / mode)
        prm = flat((33, 9, 8), nt=20)
        stage(prm, d)
        s = _lib.Solver(d, open(os.path.join(d, 'sord.in')).read())
        try:
            s.set_arithmetic(mode)
            s.step(5)
            for f, k in (('mu', 0.5), ('lam', 0.7), ('yy', 0.6)):
                s.set_field(f, k * s.field(f))
                s.step(2)
            s.step(4)
            out.append(np.concatenate([s.field('v' + a).ravel() for a in 'xyz']).astype(float))
        finally:
            s.close()
    assert np.linalg.norm(out[1] - out[0]) <= 1e-5 * np.linalg.norm(out[0])


@pytest.mark.gpu
def test_modal_step_beside_separate_steps(tmp_path, gpu_lib):
    """Steps that write stress run the separate kernels, whose stress fields
    share memory with the statics of the steps between them: twelve steps,
    stress at every third, against the run in reference order, 1e-5 of each
    quantity."""
    out = []
    for mode in ('reference', 'fast'):
        d = str(tmp_path / mode)
        prm = flat((33, 9, 8), nt=12)
        for f in ('wxx', 'wyz', 'wzx', 'wxy'):
            prm[f] = [([[], [], [], [2, None, 3]], '=>', f + '.bin')]
        stage(prm, d)
        sc.run_gpu(d, arithmetic=mode)
        w = np.concatenate([np.fromfile(os.path.join(d, f + '.bin'), '<f4') for f in ('wxx', 'wyz', 'wzx', 'wxy')])
        out.append(dict(read(d, 4), w=w.astype(float)))
    for k in out[0]:
        assert np.linalg.norm(out[1][k] - out[0][k]) <= 1e-5 * np.linalg.norm(out[0][k]), k
