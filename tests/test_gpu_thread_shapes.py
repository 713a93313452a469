"""Two host threads traverse with launch shapes of their own on two contexts: what one
sets for a kernel must not fail the other's launches."""
import threading

import pytest

import kdop_b200 as kd
from kdop_b200 import scenes

pytestmark = pytest.mark.gpu


def test_two_stack_sizes_at_once(cuda_library_path):
    sc = scenes.small_batch(n_pairs=3, seed=3)

    def posed():
        ds = kd.DeviceScene(kd.Context(0), sc.K, sc.meshes)
        ds.set_poses(sc.quat, sc.pos)
        ds.refit(kd.REFIT_POSE)
        return ds

    sides = [(posed(), {"stack_cap": 1024, "block_warps": 16}), (posed(), {"stack_cap": 64, "block_warps": 4})]
    want = sides[0][0].traverse_sync(sc.pairs).n_tests
    errors = []

    def work(ds, kw):
        opts = ds.opts(**kw)
        try:
            for _ in range(100):
                for _ in range(20):
                    ds.traverse(sc.pairs, opts)
                assert ds.stats().n_tests == want
        except BaseException as e:  # noqa: B902 -- reported by the test's own thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=side) for side in sides]
    for t in threads:
        t.start()
    for t in threads:
        t.join(120)
    assert not errors, errors
