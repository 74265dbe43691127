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
