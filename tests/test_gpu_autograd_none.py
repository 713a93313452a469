"""Gradients of a step without contacts are zero."""
import pytest

from test_gpu_autograd_streams import make

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_gradient_of_no_contacts(ctx):
    from kdop_b200.autograd import contact_geometry
    sc, ds, world = make(ctx, apart=100.0)
    x = world.clone().requires_grad_(True)
    depth, normal = contact_geometry(x, ds, sc.pairs)
    grad, = torch.autograd.grad((depth * depth).sum() + normal.sum(), x)
    assert tuple(grad.shape) == tuple(x.shape) and not grad.any()
    # with contacts again
    sc, ds, world = make(ctx)
    x = world.clone().requires_grad_(True)
    depth, normal = contact_geometry(x, ds, sc.pairs)
    grad, = torch.autograd.grad((depth * depth).sum(), x)
    assert len(depth) > 50 and grad.any()
