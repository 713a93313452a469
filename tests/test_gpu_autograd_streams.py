"""contact_geometry orders the scene's stream against torch's by events: inputs
still being written on another stream, results used at once, no contacts."""
import numpy as np
import pytest

import kdop_b200 as kd
from kdop_b200 import scenes

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def make(ctx, n_pairs=4, n=5, apart=0.0):
    sc = scenes.config5(n_pairs=n_pairs, n=n)
    sc.pos[1::2] += np.float32(apart)
    ds = kd.DeviceScene(ctx, sc.K, sc.meshes)
    ds.set_poses(sc.quat, sc.pos)
    ds.refit(kd.REFIT_POSE)
    return sc, ds, torch.from_numpy(ds.read_vertices()).cuda()


def step(x, ds, pairs):
    from kdop_b200.autograd import contact_geometry
    depth, normal = contact_geometry(x, ds, pairs)
    loss = (depth * depth).sum() + normal[:, 0].sum()
    grad, = torch.autograd.grad(loss, x)
    return depth, normal, grad


def canonical(depth, normal):
    a = torch.cat([depth[:, None], normal], 1).cpu().numpy().view(np.uint32)
    return a[np.lexsort(a.T[::-1])]


@pytest.mark.parametrize("side", [False, True])
def test_inputs_written_late_and_results_used_at_once(ctx, side):
    sc, ds, world = make(ctx)
    want = step(world.clone().requires_grad_(True), ds, sc.pairs)
    torch.cuda.synchronize()
    stream = torch.cuda.Stream() if side else torch.cuda.current_stream()
    with torch.cuda.stream(stream):
        stream.wait_stream(torch.cuda.default_stream())
        big = torch.randn(4096, 4096, device="cuda")
        for _ in range(20):
            big = big @ big * 1e-3  # keeps the stream busy before x is written
        x = (world + 0.0 * big.nan_to_num(0.0, 0.0, 0.0)[0, 0]).requires_grad_(True)
        depth, normal, grad = step(x, ds, sc.pairs)
        twice = grad + grad  # torch work on the result straight away
    stream.synchronize()
    assert len(depth) > 50
    assert np.array_equal(canonical(depth.detach(), normal.detach()), canonical(want[0].detach(), want[1].detach()))
    scale = float(want[2].abs().max())
    # float atomics add each vertex's contributions in any order: a few ulp of the largest
    assert float((grad - want[2]).abs().max()) <= 1e-5 * scale
    assert torch.equal(twice, 2 * grad)


def test_no_contacts(ctx):
    from kdop_b200.autograd import contact_geometry
    sc, ds, world = make(ctx, apart=100.0)
    depth, normal = contact_geometry(world.clone().requires_grad_(True), ds, sc.pairs)
    assert tuple(depth.shape) == (0,) and tuple(normal.shape) == (0, 3)
