"""Outputs of contact_geometry are tensors of their own for any number of
contacts, none and one included: dense, writable in place, not the contact rows'
storage."""
import numpy as np
import pytest

import kdop_b200 as kd
from kdop_b200 import scenes

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def scene_of(contacts):
    if contacts == "many":
        sc = scenes.config5(2, 3, 1, 14)
        return sc.meshes, sc.quat, sc.pos, sc.pairs
    # two tets: the apex of the second pokes through a face of the first, or hangs above it
    base = np.array([[0, 0, 0], [4, 0, 0], [0, 4, 0], [1, 1, -3]], np.float32)
    poke = np.array([[1, 1, -0.1], [0.5, 0.8, 3], [1.5, 0.8, 3], [1, 1.6, 3]], np.float32)
    meshes = []
    for x in (base, poke):
        turn = np.linalg.det((x[1:] - x[0]).astype(np.float64)) < 0
        meshes.append(scenes.Mesh(x, np.array([[0, 2, 1, 3] if turn else [0, 1, 2, 3]], np.uint32), None))
    quat = np.array([[1, 0, 0, 0]] * 2, np.float32)
    pos = np.array([[0, 0, 0], [0, 0, 0.0 if contacts == "one" else 0.5]], np.float32)
    return meshes, quat, pos, np.array([[0, 1]], np.uint32)


@pytest.mark.parametrize("contacts", ["none", "one", "many"])
def test_outputs_are_their_own(ctx, contacts):
    from kdop_b200.autograd import contact_geometry
    meshes, quat, pos, pairs = scene_of(contacts)
    ds = kd.DeviceScene(ctx, 14, meshes)
    ds.set_poses(quat, pos)
    ds.refit(kd.REFIT_POSE)
    x = torch.from_numpy(ds.read_vertices()).cuda().requires_grad_(True)
    depth, normal = contact_geometry(x, ds, pairs)
    n = len(depth)
    assert {"none": n == 0, "one": n == 1, "many": n > 1}[contacts]
    assert tuple(normal.shape) == (n, 3)
    assert depth.stride() == (1,) and normal.stride() == (3, 1)
    for out in (depth, normal):
        assert not out._is_view() and out.untyped_storage().nbytes() == 4 * out.numel()
    depth.mul_(2.0)  # refused by autograd on a view
    normal.add_(1.0)
    if n:
        grad, = torch.autograd.grad(depth.sum() + normal.sum(), x)
        assert grad.shape == x.shape and bool(grad.any())
