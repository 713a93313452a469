"""The batched traversal's seed pass (breadth-first expansion before the
persistent kernel) at the pair counts where its shape changes: one and two
passes, one and several pairs per block, pairs that end inside it and pairs
that go on.  Candidates and test counts equal the oracle's and those of the
traversal that starts from the root pairs (wave_pairs)."""
import numpy as np
import pytest

import kdop_b200 as kd
from kdop_b200 import scenes
from conftest import sorted_rows, world_xyz

pytestmark = pytest.mark.gpu


def pool_scene(n_pairs, K, sizes, seed):
    """n_pairs random pairs over a pool of overlapping lattices (some pairs
    repeat, some are far apart)."""
    rng = np.random.default_rng(seed)
    meshes = [scenes.lattice(int(n), 0.15, rng) for n in sizes]
    quat = np.stack([scenes.random_quaternion(rng) for _ in sizes])
    pos = rng.uniform(-2.0, 2.0, (len(sizes), 3)).astype(np.float32)
    pos[-1] += 100.0  # a body that overlaps nothing
    pairs = rng.integers(0, len(sizes), (n_pairs, 2)).astype(np.uint32)
    return scenes.Scene("pool", K, meshes, quat, pos, pairs)


@pytest.mark.parametrize("n_pairs,K,sizes", [(1, 14, (10, 10)), (1, 26, (1, 1)), (63, 6, (1, 2, 5, 3)),
                                             (64, 18, (4, 6, 2)), (65, 20, (4, 6, 2)), (593, 8, (1, 3, 4, 2)),
                                             (1185, 12, (2, 1, 3))])
@pytest.mark.parametrize("surface_filter", [1, 0])
def test_seeded_traversal_equals_the_root_traversal_and_the_oracle(ctx, oracle, n_pairs, K, sizes, surface_filter):
    sc = pool_scene(n_pairs, K, sizes, 31 + n_pairs)
    if n_pairs == 1:
        sc.pairs[:] = (0, 1)
        sc.pos[:] = 0.25 * np.arange(2)[:, None]
    ds = kd.DeviceScene(ctx, sc.K, sc.meshes)
    ds.set_poses(sc.quat, sc.pos)
    ds.refit(kd.REFIT_POSE)
    seeded = ds.traverse_sync(sc.pairs, ds.opts(surface_filter=surface_filter))
    got = sorted_rows(ds.candidates())
    roots = ds.traverse_sync(sc.pairs, ds.opts(surface_filter=surface_filter, wave_pairs=n_pairs))
    assert np.array_equal(got, sorted_rows(ds.candidates()))
    assert (seeded.n_tests, seeded.n_leaf_overlaps) == (roots.n_tests, roots.n_leaf_overlaps)
    worlds = [world_xyz(oracle, sc, i) for i in range(len(sc.meshes))]
    want, tests, _ = oracle.run_pairs(sc.K, worlds, sc.meshes, sc.pairs)
    assert seeded.n_tests == int(np.sum(tests))
    if surface_filter:
        assert np.array_equal(got, sorted_rows(want))
    else:
        assert len(got) == seeded.n_leaf_overlaps
