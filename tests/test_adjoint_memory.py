"""A gradient whose backward pass has run is returned whatever is left of
the device memory."""
import numpy as np
import pytest


@pytest.mark.gpu
def test_material_chain_without_device_memory(monkeypatch, gpu_lib):
    """The library has no memory for the material chain rule: the same
    gradients from the host; its other errors are raised."""
    import torch
    from coseis_b200 import _lib, adjoint
    n, nt = (16, 14, 12), 12
    prm = {'shape': list(n) + [nt], 'delta': [100.0, 90.0, 110.0, 0.005], 'bc1': ['free'] * 3, 'bc2': ['free'] * 3,
           'npml': 0, 'hourglass': [1.0, 0.5], 'gam': [0.0], 'itstats': 10, 'itio': 20}
    p = adjoint.Problem(prm, {'x': [7.5, 6.5, 5.5], 'pulse': 'ricker2', 'tau': 0.05}, [[4.0, 5.0, 3.0]], segment=1)
    rng = np.random.default_rng(4)
    cells = tuple(x - 1 for x in n)
    vals = [(v * (1 + 0.05 * rng.random(cells))).astype('f4') for v in (2700.0, 6000.0, 3464.0)]
    seen = torch.from_numpy(rng.standard_normal((1, 3, nt)).astype('f4'))

    def gradients():
        v = [torch.from_numpy(a).requires_grad_() for a in vals]
        tr = adjoint.ReceiverTraces.apply(*v, torch.full((6,), 1e15, dtype=torch.float64), p)
        (tr * seen).sum().backward()
        return [a.grad.numpy() for a in v]

    def refuse(code):
        def call(self, *a):
            raise _lib.SordError(code, 'refused')
        monkeypatch.setattr(_lib.Solver, 'adjoint_material', call)

    want = gradients()
    assert all(np.abs(a).max() > 0 for a in want)
    refuse(_lib.SORD_E_NOMEM)
    for a, b in zip(gradients(), want):
        assert np.array_equal(a, b)
    refuse(_lib.SORD_E_CUDA)
    with pytest.raises(_lib.SordError):
        gradients()
