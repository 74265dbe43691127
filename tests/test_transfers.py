"""What crosses between device and host in batches: fields in chunks of planes
(sord_get_field, sord_set_field), the outputs that fire together in one launch,
and the material chain rule of the gradients in slabs of rows.  Each moves or
repeats values exactly, so every comparison is of bits."""
import os

import numpy as np
import pytest

import sordcases as sc


def solver(prm, path):
    from coseis_b200 import _lib
    sc.stage(prm, path)
    return _lib.Solver(path, open(os.path.join(path, 'sord.in')).read())


@pytest.mark.gpu
@pytest.mark.parametrize('shape', [(7, 5, 9), (33, 2, 40), (165, 163, 170), (230, 220, 210)],
                         ids=['small', 'thin', '2-chunks', '3-chunks'])
def test_field_round_trip(shape, tmp_path, gpu_lib):
    prm = {'shape': list(shape) + [2], 'delta': [100.0, 100.0, 100.0, 0.0075], 'rho': [2670.0], 'vp': [6000.0],
           'vs': [3464.0], 'bc1': ['free'] * 3, 'bc2': ['free'] * 3, 'npml': 0, 'itio': 2}
    s = solver(prm, str(tmp_path))
    try:
        rng = np.random.default_rng(5)
        before = {f: s.field(f).copy() for f in ('vy', 'mu', 'uz')}
        for f, n in (('vx', shape), ('lam', tuple(x - 1 for x in shape))):
            a = rng.standard_normal(s.field(f).shape, dtype=np.float32)
            assert sorted(a.shape) == sorted(n)
            s.set_field(f, a)
            assert np.array_equal(s.field(f), a), f
        for f, a in before.items():
            assert np.array_equal(s.field(f), a), f
    finally:
        s.close()


@pytest.mark.gpu
@pytest.mark.parametrize('stress', [False, True], ids=['one-kernel', 'separate'])
def test_outputs_fire_together(stress, tmp_path, gpu_lib):
    """More probes and gathers in a step than a batch holds, of several
    fields, and buffers that fill in mid-run, against whole-volume records."""
    n, nt = (14, 12, 10), 4
    prm = {'shape': list(n) + [nt], 'delta': [100.0, 100.0, 100.0, 0.0075], 'rho': [2670.0], 'vp': [6000.0],
           'vs': [3464.0], 'hourglass': [1.0, 1.0], 'bc1': ['pml'] * 3, 'bc2': ['pml'] * 3, 'npml': 3, 'itio': 2,
           'mxy': [([6.5, 5.5, 4.5, []], '.', 1e14, 'ricker1', 0.02)]}
    rng = np.random.default_rng(9)
    at = [[int(rng.integers(1, m - 1)) for m in n] for _ in range(50)]
    fields = ['vx', 'vy', 'vz'] + (['wxx', 'wyy', 'wzz', 'wyz', 'wzx', 'wxy'] if stress else [])
    for f in fields:
        prm[f] = [([[], [], [], []], '=>', 'all-%s.bin' % f)]
        prm[f] += [(p + [[]], '=>', 'g%02d-%s.bin' % (i, f)) for i, p in enumerate(at[:13])]
        if f[0] == 'v':
            prm[f] += [(p + [[]], '.>', 'p%02d-%s.bin' % (i, f)) for i, p in enumerate(at)]
    d = str(tmp_path)
    s = solver(prm, d)
    try:
        s.run()
    finally:
        s.close()
    read = lambda name: np.fromfile(os.path.join(d, name), '<f4')
    for f in fields:
        m = n if f[0] == 'v' else tuple(x - 1 for x in n)
        whole = read('all-%s.bin' % f).reshape((nt,) + m[::-1])
        assert np.abs(whole).max() > 0
        for i, (j, k, l) in enumerate(at):
            if i < 13:
                assert np.array_equal(read('g%02d-%s.bin' % (i, f)), whole[:, l, k, j]), (f, i)
            if f[0] == 'v':
                assert np.array_equal(read('p%02d-%s.bin' % (i, f)), whole[:, l, k, j]), (f, i)


@pytest.mark.gpu
@pytest.mark.parametrize('shape', [(18, 16, 14), (5, 33, 9), (4, 1450, 1450)], ids=['small', 'ragged', '3-slabs'])
def test_material_chain_on_device(shape, tmp_path, gpu_lib):
    """Solver.adjoint_material against adjoint.material_chain, with cells of
    no mass and no modulus among them."""
    from coseis_b200 import _lib, adjoint
    delta = [100.0, 80.0, 120.0]
    prm = {'shape': list(shape) + [3], 'delta': delta + [0.005], 'bc1': ['free'] * 3, 'bc2': ['free'] * 3, 'npml': 0,
           'hourglass': [1.0, 0.5], 'gam': [0.0], 'itstats': 10, 'itio': 20}
    c = [0.5 * (x - 1) for x in shape]
    p = adjoint.Problem(prm, {'x': c, 'pulse': 'ricker2', 'tau': 0.05}, [[float(int(x)) for x in c]], segment=1)
    nc = tuple(x - 1 for x in shape)
    rng = np.random.default_rng(3)
    vals = [v * (1 + 0.05 * rng.random(nc, dtype=np.float32)) for v in (2700.0, 6000.0, 3464.0)]
    d = str(tmp_path)
    files = p.stage(*vals, [1e15] * 6, d)
    s = _lib.Solver(d, open(os.path.join(d, 'sord.in')).read())
    try:
        p.forward(s)
        g = s.adjoint_backward({f: rng.standard_normal(3).astype(np.float32) for f in files}, 6)
        assert np.abs(g['lam']).max() > 0
        vals[0][0, 0, 0] = 0.0
        vals[0][-1] = 0.0
        vals[2][1, 1] = 0.0
        for a, b in zip(s.adjoint_material(*vals, delta), adjoint.material_chain(*vals, g, delta)):
            assert np.array_equal(a, b)
    finally:
        s.close()
