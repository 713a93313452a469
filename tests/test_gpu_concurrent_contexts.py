"""Traversals that share the GPU: two contexts traverse from two host threads,
each launch sized for the whole GPU, so that blocks of one wait for places the
other holds.  A launch must finish with whatever part of its blocks runs."""
import threading

import numpy as np
import pytest

import kdop_b200 as kd
from kdop_b200 import scenes
from conftest import sorted_rows

pytestmark = pytest.mark.gpu


# frontiers of both seed passes (up to 64 pairs) and of one
@pytest.mark.parametrize("n_pairs", [2, 96])
def test_two_contexts_traverse_at_once(cuda_library_path, n_pairs):
    def posed(seed):
        own = kd.Context(0)
        sc = scenes.config3(n_pairs, seed, 4000, 40000, 0.15, 14)
        ds = kd.DeviceScene(own, sc.K, sc.meshes)
        ds.set_poses(sc.quat, sc.pos)
        ds.refit(kd.REFIT_POSE)
        st = ds.traverse_sync(sc.pairs)
        return ds, sc.pairs, st, sorted_rows(ds.candidates())

    sides = [posed(seed) for seed in (1, 2)]
    start = threading.Barrier(2)
    errors = []

    def work(ds, pairs, want, rows):
        try:
            start.wait(30)
            for _ in range(20):
                for _ in range(4):
                    ds.traverse(pairs)
                st = ds.stats()  # raises on a wait that timed out
                assert (st.n_tests, st.n_candidates) == (want.n_tests, want.n_candidates)
            assert np.array_equal(sorted_rows(ds.candidates()), rows)
        except BaseException as e:  # noqa: B902 -- reported by the test's own thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=side) for side in sides]
    for t in threads:
        t.start()
    for t in threads:
        t.join(120)
    assert not errors, errors
