"""Point sources inside the step kernels."""
import os

import numpy as np
import pytest

import sordcases as sc

MOMENT = ('mxx', 'myy', 'mzz', 'myz', 'mzx', 'mxy')


def hill(n, dx):
    """z of a terrain mesh [j, k, l]."""
    x, y, z = np.meshgrid(*[np.arange(m) for m in n], indexing='ij')
    top = 3.0 * dx * np.exp(-((x - n[0] / 2.0) ** 2 + (y - n[1] / 2.0) ** 2) / (2.0 * (n[1] / 6.0) ** 2))
    return dx * z - top * (1.0 - z / (n[2] - 1.0))


@pytest.mark.gpu
@pytest.mark.parametrize('arithmetic', ['reference', 'fast'])
def test_sources_far_apart_cost_little(arithmetic, tmp_path, gpu_lib):
    """Each block of a step kernel takes the sources in its own box: four
    moment sources far apart may take half as long again as one (a block that
    takes the others' too: 2.6 times in fast arithmetic)."""
    from coseis_b200 import _lib
    n, dx = (256, 256, 128), 50.0
    near = [[128.25, 128.25, 64.25]]
    far = [[x, y, 38.65 if x < 128 else 89.85] for x in (77.05, 179.45) for y in (77.05, 179.45)]
    z = hill(n, dx).astype('<f4').ravel(order='F')
    took = []
    for name, at in (('near', near), ('far', far)):
        d = str(tmp_path / name)
        os.makedirs(d)
        z.tofile(os.path.join(d, 'z.bin'))
        prm = {'shape': list(n) + [10 ** 6], 'delta': [dx] * 3 + [0.004], 'rho': [2670.0], 'vp': [6000.0],
               'vs': [3464.0], 'gam': [0.1], 'hourglass': [1.0, 1.0], 'bc1': ['pml', 'pml', 'free'],
               'bc2': ['pml'] * 3, 'npml': 12, 'itstats': 10 ** 6, 'itio': 10 ** 6, 'z': [([], '=<', 'z.bin')]}
        for i, f in enumerate(MOMENT):
            prm[f] = [(x + [[]], '.', 1e14 * (i - 2.5), 'brune', 0.1) for x in at]
        sc.stage(prm, d)
        s = _lib.Solver(d, open(os.path.join(d, 'sord.in')).read())
        try:
            s.set_arithmetic(arithmetic)
            s.step(3)
            ms = []
            for _ in range(5):
                s.step(10)
                ms.append(s.last_step_ms())
            assert np.isfinite(s.field('vx')).all()
        finally:
            s.close()
        took.append(min(ms))
    assert took[1] <= 1.5 * took[0], took


def crowded(n, mesh, path, realsize=4):
    """Ten full tensors: in one interior tile, and in one box of the PML
    shell, more entries (two moment tensors, 96; two potency tensors, 96) than
    a block keeps (64), and one of each far from both."""
    at = [[n[0] / 2.0 + 0.3, n[1] / 2.0 - 0.2, n[2] / 2.0 + 0.1], [n[0] / 2.0 + 2.7, n[1] / 2.0 + 0.4, n[2] / 2.0 - 0.6],
          [1.5, n[1] / 2.0, n[2] / 2.0], [2.25, n[1] / 2.0 + 1.5, n[2] / 2.0 + 0.5], [n[0] - 7.5, n[1] - 7.25, 5.5]]
    prm = {'shape': list(n) + [10], 'delta': [100.0, 100.0, 100.0, 0.008], 'rho': [2670.0], 'vp': [6000.0],
           'vs': [3464.0], 'gam': [0.2], 'hourglass': [1.0, 2.0], 'bc1': ['pml', 'pml', 'free'], 'bc2': ['pml'] * 3,
           'npml': 4, 'vpml': 4000.0, 'itstats': 3, 'itio': 10}
    for i, f in enumerate(MOMENT):
        prm[f] = [(x + [[]], '.', 1e15 * (i - 2.5) * (1 + s), 'brune', 0.05) for s, x in enumerate(at)]
        prm['p' + f[1:]] = [(x + [[]], '.', 3e4 * (i - 1.5) * (1 + s), 'brune', 0.05) for s, x in enumerate(at)]
    for f in ('vx', 'vy', 'vz', 'ux', 'uy', 'uz'):
        prm[f] = [([[], [], [], -1], '=>', 'vol-%s.bin' % f)]
    os.makedirs(path)
    j, k, l = np.meshgrid(*[np.arange(m) for m in n], indexing='ij')
    x = {'z': 100.0 * l - 40.0 * np.sin(j / 3.0) * np.cos(k / 4.0) * (1.0 - l / (n[2] - 1.0)),
         'x': 100.0 * j + 15.0 * np.sin(k / 3.0) * np.cos(l / 4.0)}
    for f in {'flat': '', 'terrain': 'z', 'general': 'xz'}[mesh]:
        x[f].astype('<f%d' % realsize).ravel(order='F').tofile(os.path.join(path, f + '.bin'))
        prm[f] = [([], '=<', f + '.bin')]
    sc.stage(prm, path, realsize=realsize)


def volumes(path, size):
    f = lambda q: np.concatenate([np.fromfile(os.path.join(path, 'vol-%s%s.bin' % (q, a)), '<f%d' % size) for a in 'xyz'])
    return {q: f(q).astype(float) for q in 'vu'}


@pytest.mark.gpu
@pytest.mark.parametrize('mesh', ['flat', 'terrain', 'general'])
def test_more_sources_than_a_block_keeps(mesh, tmp_path, oracle_bins, gpu_lib):
    """Reference order: the bits of the FP32 oracle.  Fast arithmetic: within
    twice that oracle's error against the FP64 one, or 1e-6, and other bits."""
    d = {k: str(tmp_path / k) for k in ('o64', 'o32', 'reference', 'fast')}
    for k, path in d.items():
        crowded((43, 26, 24), mesh, path, 8 if k == 'o64' else 4)
    sc.run_oracle(d['o64'], oracle_bins['f64'])
    sc.run_oracle(d['o32'], oracle_bins['f32'])
    for mode in ('reference', 'fast'):
        sc.run_gpu(d[mode], arithmetic=mode)
    b, c = volumes(d['o64'], 8), volumes(d['o32'], 4)
    ref, fast = volumes(d['reference'], 4), volumes(d['fast'], 4)
    for q in 'vu':
        n = np.linalg.norm(b[q])
        assert n > 0 and np.isfinite(n)
        assert np.array_equal(ref[q], c[q]), q
        e, e32 = np.linalg.norm(fast[q] - b[q]) / n, np.linalg.norm(c[q] - b[q]) / n
        assert e <= max(2 * e32, 1e-6), (q, e, e32)
        assert not np.array_equal(fast[q], c[q])
