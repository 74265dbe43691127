"""The meshes and options of tests/test_modal_step.py that the corner-mode
kernel takes, held closer: its rounding is that of an FP32 run, so its error
against the FP64 oracle is at most twice the FP32 oracle's, or 1e-6; and its
bits are not those of the reference order, so it is the kernel that ran."""
import numpy as np
import pytest

import sordcases as sc
import test_modal_step as modal


@pytest.mark.gpu
@pytest.mark.parametrize('name', sorted(set(modal.CASES) - {'sheared'}))
def test_modal_accuracy(name, tmp_path, oracle_bins, gpu_lib):
    prm = modal.CASES[name]()
    d = {k: str(tmp_path / k) for k in ('o64', 'o32', 'fast')}
    for k, path in d.items():
        modal.stage(prm, path, 8 if k == 'o64' else 4)
    sc.run_oracle(d['o64'], oracle_bins['f64'])
    sc.run_oracle(d['o32'], oracle_bins['f32'])
    sc.run_gpu(d['fast'], arithmetic='fast')
    a, b, c = modal.read(d['fast'], 4), modal.read(d['o64'], 8), modal.read(d['o32'], 4)
    assert sorted(a) == ['u', 'v']
    for q in a:
        n = np.linalg.norm(b[q])
        e, e32 = np.linalg.norm(a[q] - b[q]) / n, np.linalg.norm(c[q] - b[q]) / n
        assert e <= max(2 * e32, 1e-6), (q, e, e32)
        assert not np.array_equal(a[q], c[q]), q
