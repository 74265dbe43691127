"""Device memory that stays in the pool after a handle is destroyed."""
import os
import time

import pytest

import sordcases as sc


def handle(path, n):
    from coseis_b200 import _lib
    prm = {'shape': [n, n, n, 2], 'delta': [100.0, 100.0, 100.0, 0.0075], 'rho': [2670.0], 'vp': [6000.0],
           'vs': [3464.0], 'bc1': ['free'] * 3, 'bc2': ['free'] * 3, 'npml': 0, 'itio': 2}
    sc.stage(prm, path)
    return _lib.Solver(path, open(os.path.join(path, 'sord.in')).read())


@pytest.mark.gpu
def test_memory_goes_back_without_a_call(tmp_path, monkeypatch, gpu_lib):
    """The fields of a closed handle (1.4 GB) serve the next one, and go back
    to the driver by themselves when none comes (within SORD_POOL_IDLE
    seconds); sord_trim_memory returns them at once."""
    import torch
    from coseis_b200 import _lib
    monkeypatch.setenv('SORD_POOL_IDLE', '4')
    free = lambda: torch.cuda.mem_get_info()[0]
    handle(str(tmp_path / 'first'), 220).close()  # what a first handle loads stays
    _lib.trim_memory(0)
    before, small = free(), 100 << 20
    for i in range(2):
        s = handle(str(tmp_path / str(i)), 220)
        assert before - free() > (1 << 30)
        s.close()
    end = time.time() + 30
    while before - free() > small and time.time() < end:
        time.sleep(0.5)
    assert before - free() <= small
    handle(str(tmp_path / 'last'), 220).close()
    _lib.trim_memory(0)
    assert before - free() <= small
