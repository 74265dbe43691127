"""Fast arithmetic with a negative viscous hourglass constant, which the
reference applies outside the PML only (acceleration.f90:164): the interior in
corner modes, the shell in reference order."""
import os

import numpy as np
import pytest

import sordcases as sc

HOURGLASS = [1.0, -0.02]


def model(n, nt, mesh, path, realsize=4):
    c = [m / 2.0 - 0.2 for m in n]
    prm = {'shape': list(n) + [nt], 'delta': [100.0, 100.0, 100.0, 0.008], 'rho': [2670.0], 'vp': [6000.0],
           'vs': [3464.0], 'gam': [0.2], 'hourglass': HOURGLASS, 'bc1': ['pml', 'pml', 'free'], 'bc2': ['pml'] * 3,
           'npml': 4, 'vpml': 4000.0, 'itstats': 3, 'itio': 10, 'mxx': [(c + [[]], '.', 1e15, 'brune', 0.05)],
           'myz': [(c + [[]], '.', -4e14, 'brune', 0.05), ([2.5, c[1], c[2], []], '.', 1e14, 'brune', 0.05)]}
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


def read(path, size):
    f = lambda q: np.concatenate([np.fromfile(os.path.join(path, 'vol-%s%s.bin' % (q, a)), '<f%d' % size) for a in 'xyz'])
    return {q: f(q).astype(float) for q in 'vu'}


@pytest.mark.gpu
@pytest.mark.parametrize('mesh', ['flat', 'terrain', 'general'])
def test_accuracy(mesh, tmp_path, oracle_bins, gpu_lib):
    """Within twice the FP32 oracle's error against the FP64 oracle, or 1e-6;
    not the bits of the reference order, so the fast kernels ran."""
    d = {k: str(tmp_path / k) for k in ('o64', 'o32', 'fast')}
    for k, path in d.items():
        model((43, 19, 18), 10, mesh, path, 8 if k == 'o64' else 4)
    sc.run_oracle(d['o64'], oracle_bins['f64'])
    sc.run_oracle(d['o32'], oracle_bins['f32'])
    sc.run_gpu(d['fast'], arithmetic='fast')
    a, b, c = read(d['fast'], 4), read(d['o64'], 8), read(d['o32'], 4)
    for q in 'vu':
        n = np.linalg.norm(b[q])
        assert n > 0 and np.isfinite(n)
        e, e32 = np.linalg.norm(a[q] - b[q]) / n, np.linalg.norm(c[q] - b[q]) / n
        assert e <= max(2 * e32, 1e-6), (q, e, e32)
        assert not np.array_equal(a[q], c[q])


@pytest.mark.gpu
def test_no_slower_than_reference_order(tmp_path, gpu_lib):
    from coseis_b200 import _lib
    d = str(tmp_path / 'm')
    model((300, 150, 150), 10 ** 6, 'flat', d)
    s = _lib.Solver(d, open(os.path.join(d, 'sord.in')).read())
    best = {}
    try:
        for mode in ('reference', 'fast'):
            s.set_arithmetic(mode)
            s.step(2)
            for _ in range(5):
                s.step(5)
                best[mode] = min(best.get(mode, 1e9), s.last_step_ms())
    finally:
        s.close()
    assert best['fast'] <= best['reference'], best
