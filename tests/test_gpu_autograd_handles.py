"""contact_geometry with a context on a stream of the caller's, the special handles
of the default streams (1: legacy, 2: per thread) among them."""
import pytest

import kdop_b200 as kd
from test_gpu_autograd_streams import canonical, make, step

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("handle", [1, 2, None])
def test_stream_handles(ctx, handle):
    sc, ds, world = make(ctx)
    want = step(world.clone().requires_grad_(True), ds, sc.pairs)
    stream = torch.cuda.Stream()
    own = kd.Context(0, stream=handle or stream.cuda_stream)
    sc, ds, world = make(own)
    got = step(world.clone().requires_grad_(True), ds, sc.pairs)
    torch.cuda.synchronize()
    assert len(got[0]) > 50
    assert (canonical(got[0].detach(), got[1].detach()) == canonical(want[0].detach(), want[1].detach())).all()
    # float atomics add each vertex's contributions in any order: a few ulp of the largest
    assert float((got[2] - want[2]).abs().max()) <= 1e-5 * float(want[2].abs().max())
