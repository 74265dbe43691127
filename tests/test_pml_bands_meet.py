"""Decks whose PML bands of opposite faces share cells (the front end refuses
them): such a cell or node is damped by both, the near face first."""
import os

import numpy as np
import pytest

import sordcases as sc

# shape, npml of the deck: x bands share one cell layer; cells and nodes of x;
# one layer of every axis
MESHES = {'x': ((10, 34, 30), 5), 'x_nodes': ((10, 34, 30), 6), 'xyz': ((10, 10, 10), 5)}


def stage(path, shape, npml, mesh, realsize=4):
    """A deck staged with thinner bands, which are then widened in its text."""
    n = list(shape)
    c = [m / 2.0 - 0.2 for m in n]
    prm = {'shape': n + [12], 'delta': [100.0, 100.0, 100.0, 0.008], 'rho': [2670.0], 'vp': [6000.0], 'vs': [3464.0],
           'gam': [0.1], 'hourglass': [1.0, 1.0], 'bc1': ['pml'] * 3, 'bc2': ['pml'] * 3, 'npml': 3, 'vpml': 4000.0,
           'itstats': 3, 'itio': 12, 'mxx': [(c + [[]], '.', 1e15, 'brune', 0.05)],
           'myz': [(c + [[]], '.', -4e14, 'brune', 0.05)]}
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
    deck = os.path.join(path, 'sord.in')
    first, rest = open(deck).read().split('\n', 1)
    t = first.split()
    # the values of the sorted keys: i1pml, i2pml and npml
    assert t[30:36] == ['3'] * 3 + [str(m - 3) for m in n] and t[47] == '3'
    t[30:36] = [str(npml)] * 3 + [str(m - npml) for m in n]
    t[47] = str(npml)
    with open(deck, 'w') as fh:
        fh.write(' '.join(t) + '\n' + rest)


def read(path, size):
    f = lambda q: np.concatenate([np.fromfile(os.path.join(path, 'vol-%s%s.bin' % (q, a)), '<f%d' % size) for a in 'xyz'])
    return {q: f(q).astype(float) for q in 'vu'}


@pytest.mark.gpu
@pytest.mark.parametrize('mesh', ['flat', 'terrain', 'general'])
@pytest.mark.parametrize('name', sorted(MESHES))
def test_bands_meet(name, mesh, tmp_path, oracle_bins, gpu_lib):
    """Both arithmetics against the oracle: reference order bit for bit, fast
    within ten times the FP32 oracle's error against the FP64 one, or 1e-6."""
    shape, npml = MESHES[name]
    d = {k: str(tmp_path / k) for k in ('o64', 'o32', 'reference', 'fast')}
    for k, path in d.items():
        stage(path, shape, npml, mesh, 8 if k == 'o64' else 4)
    sc.run_oracle(d['o64'], oracle_bins['f64'])
    sc.run_oracle(d['o32'], oracle_bins['f32'])
    for mode in ('reference', 'fast'):
        sc.run_gpu(d[mode], arithmetic=mode)
    b, c = read(d['o64'], 8), read(d['o32'], 4)
    ref, fast = read(d['reference'], 4), read(d['fast'], 4)
    for q in 'vu':
        n = np.linalg.norm(b[q])
        assert n > 0 and np.isfinite(n)
        assert np.array_equal(ref[q], c[q]), q
        e, e32 = np.linalg.norm(fast[q] - b[q]) / n, np.linalg.norm(c[q] - b[q]) / n
        assert e <= max(10 * e32, 1e-6), (q, e, e32)
