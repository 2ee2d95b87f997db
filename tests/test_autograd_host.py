"""The autograd layers' handling of shapes and gradient tensors, on the CPU: the kernel calls are
replaced by stand-ins that leave every output as allocated."""
import pytest
import torch

from geepee_gb300 import autograd, gpk


@pytest.fixture
def no_kernels(monkeypatch):
    def fill(*args, **kw):
        for t in list(args) + list(kw.values()):
            if isinstance(t, torch.Tensor) and not t.requires_grad:
                t.fill_(1.0)
    for name in ('psi_fwd', 'det_fwd', 'psi_layer_bwd', 'det_layer_bwd'):
        monkeypatch.setattr(gpk, name, fill)
    monkeypatch.setattr(gpk, 'work_elems', lambda *a: 16)


def _leaves(layer, shape, dtype):
    N, M, Q, D = 7, 5, 3, 2
    t = lambda *s: torch.rand(*s, dtype=dtype)
    rows = [t(N, Q), t(N, Q)] if layer == 'psi' else [t(N, Q)]
    ins = rows + [t(M, Q), torch.zeros(shape, dtype=dtype), torch.zeros(1, dtype=dtype), t(D, M), t(D, M, M)]
    return [a.requires_grad_(True) for a in ins]


@pytest.mark.parametrize('dtype', [torch.float64, torch.float32])
@pytest.mark.parametrize('layer', ['psi', 'det'])
@pytest.mark.parametrize('shape', [(3,), (1, 3), (3, 1)])
def test_lengthscale_gradient_has_its_shape(no_kernels, layer, shape, dtype):
    """A log-lengthscale parameter of any shape with Q entries gets a gradient of that shape."""
    ins = _leaves(layer, shape, dtype)
    m, v = getattr(autograd, layer + '_moments')(*ins)
    (m + v).sum().backward()
    for a in ins:
        assert a.grad.shape == a.shape and a.grad.dtype == a.dtype


@pytest.mark.parametrize('dtype', [torch.float64, torch.float32])
@pytest.mark.parametrize('layer', ['psi', 'det'])
def test_gradients_are_tensors_of_their_own(no_kernels, layer, dtype):
    """No gradient is a view: each can be detached in place, is aligned as an allocation is, and keeps
    no other gradient's memory."""
    ins = _leaves(layer, (3,), dtype)
    m, v = getattr(autograd, layer + '_moments')(*ins)
    (m + v).sum().backward()
    held = set()
    for a in ins:
        a.grad.detach_()
        assert a.grad.untyped_storage().nbytes() == a.grad.nbytes
        held.add(a.grad.untyped_storage().data_ptr())
    assert len(held) == len(ins)
