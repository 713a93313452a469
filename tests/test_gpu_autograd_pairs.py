"""contact_geometry with a pair list that torch converts first (64-bit, in device
memory): the scene's stream waits for the conversion, however late it runs."""
import numpy as np
import pytest

import kdop_b200 as kd
from kdop_b200 import scenes

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_pairs", [4, 300])
def test_converted_pairs(ctx, monkeypatch, n_pairs):
    from kdop_b200.autograd import contact_geometry
    sc = scenes.config5(4, 4, 1, 14)
    ds = kd.DeviceScene(ctx, sc.K, sc.meshes)
    ds.set_poses(sc.quat, sc.pos)
    ds.refit(kd.REFIT_POSE)
    world = torch.from_numpy(ds.read_vertices()).cuda()
    pairs = np.tile(sc.pairs, (n_pairs // 4, 1))
    want = len(contact_geometry(world.clone().requires_grad_(True), ds, pairs)[0])
    convert = kd.lib._arg

    def late(a, dtype):
        if hasattr(a, "is_cuda") and a.is_cuda and a.dtype == torch.int64:
            torch.cuda._sleep(40_000_000)  # about 20 ms of the current stream
        return convert(a, dtype)

    wide = torch.from_numpy(pairs.astype(np.int64)).cuda()
    torch.cuda.synchronize()
    monkeypatch.setattr(kd.lib, "_arg", late)
    depth, _ = contact_geometry(world.requires_grad_(True), ds, wide)
    assert len(depth) == want > 0
