"""Every launch shape at every K over pairs whose leaves all overlap, so that the lanes
emit as many rows a step as they can hold."""
import numpy as np
import pytest

import kdop_b200 as kd
from conftest import sorted_rows
from kdop_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [6, 8, 12, 14, 18, 20, 26])
@pytest.mark.parametrize("load_group", [1, 2, 4, 8])
def test_all_leaves_overlap(ctx, oracle, K, load_group):
    rng = np.random.default_rng(K)
    meshes = []
    for n in (6, 60, 200, 333):  # tets far apart in a lattice: nearly all have boundary faces
        whole = scenes.lattice(5, 0.1, rng)
        tets = whole.tets[np.sort(rng.permutation(whole.n_tets)[:n])]
        meshes.append(scenes.Mesh(whole.xyz, tets, scenes.surface_map(tets)))
    moved = [(m.xyz * np.float32(1e-30)).astype(np.float32) for m in meshes]  # every slab overlaps every other
    ds = kd.DeviceScene(ctx, K, meshes)
    ds.set_vertices(np.concatenate(moved))
    ds.refit(kd.REFIT_VERTICES)
    pairs = np.array([[0, 1], [2, 3], [3, 2], [1, 2], [0, 0], [2, 2]] * 2, np.uint32)
    want, tests = [], 0
    for p, (a, b) in enumerate(pairs):
        rows, n, _ = oracle.run_pair(K, moved[a], meshes[a].tets, meshes[a].surf, moved[b], meshes[b].tets,
                                     meshes[b].surf, restA=meshes[a].xyz, restB=meshes[b].xyz)
        want.append(np.column_stack([np.full(len(rows), p), rows]))
        tests += n
    want = sorted_rows(np.concatenate(want).astype(np.int64))
    for kw in ({}, {"init_chunk": 32}, {"wave_pairs": 3, "init_chunk": 1}, {"wave_pairs": 12, "init_chunk": 32},
               {"mode": kd.TRAVERSE_PLAIN}, {"stack_cap": 64, "donate_min": 1}):
        st = ds.traverse_sync(pairs, ds.opts(load_group=load_group, **kw))
        assert st.n_tests == tests, kw
        assert np.array_equal(sorted_rows(ds.candidates().astype(np.int64)), want), kw
    share = []
    for rank in range(2):
        ds.traverse_shard(pairs, rank, 2, opts=ds.opts(load_group=load_group))
        share.append(ds.candidates().astype(np.int64))
    assert np.array_equal(sorted_rows(np.concatenate(share)), want)
    ds.close()
