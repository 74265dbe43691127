"""Outputs against the inputs that follow them in the same step."""
import os

import numpy as np
import pytest

import sordcases as sc


@pytest.mark.gpu
def test_outputs_before_an_input_that_fails(tmp_path, gpu_lib):
    """The velocity records of four steps fill at the fourth, in which the
    next component's input file turns out to be missing: the step fails, the
    records are on disk as in a run without that input."""
    from coseis_b200 import _lib
    n = (9, 8, 7)
    records = []
    for broken in (False, True):
        d = str(tmp_path / str(broken))
        prm = {'shape': list(n) + [8], 'delta': [100.0, 100.0, 100.0, 0.0075], 'rho': [2670.0], 'vp': [6000.0],
               'vs': [3464.0], 'hourglass': [1.0, 1.0], 'bc1': ['free'] * 3, 'bc2': ['free'] * 3, 'npml': 0,
               'itio': 100, 'mxy': [([4.5, 4.0, 3.5, []], '.', 1e14, 'ricker1', 0.02)],
               'vx': [([[], [], [], [0, 4, 1]], '=>', 'vx.bin')]}
        if broken:
            prm['vy'] = [([[], [], [], [3, 4, 1]], '=<', 'nowhere.bin')]
        sc.stage(prm, d)
        s = _lib.Solver(d, open(os.path.join(d, 'sord.in')).read())
        try:
            if broken:
                with pytest.raises(_lib.SordError) as e:
                    s.step(8)
                assert e.value.code == _lib.SORD_E_IO
            else:
                s.step(8)
        finally:
            s.close()
        records.append(np.fromfile(os.path.join(d, 'vx.bin'), '<f4'))
    assert records[0].size == 4 * np.prod(n) and np.abs(records[0]).max() > 0
    assert np.array_equal(*records)
