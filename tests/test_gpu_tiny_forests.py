"""Refit of forests of small trees: up to 63 tets a block of one warp takes a tree,
from 64 on blocks of eight warps take them all."""
import numpy as np
import pytest

import kdop_b200 as kd
from kdop_b200 import scenes
from test_gpu_read_staging import preorder

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [6, 8, 12, 14, 18, 20, 26])
@pytest.mark.parametrize("sizes", [(1,), (1, 2), (5, 0, 63, 31, 32, 33, 1), (63, 64, 1), tuple(range(64)) * 35])
def test_forest(ctx, oracle, K, sizes):
    rng = np.random.default_rng(len(sizes))
    whole = scenes.lattice(3, 0.1, rng)
    meshes = [scenes.Mesh(whole.xyz, whole.tets[:n], scenes.surface_map(whole.tets[:n])) if n else
              scenes.Mesh(np.zeros((0, 3), np.float32), np.zeros((0, 4), np.uint32), np.zeros(0, np.uint8))
              for n in sizes]
    ds = kd.DeviceScene(ctx, K, meshes)
    moved = [(m.xyz + rng.normal(size=(1, 3))).astype(np.float32) for m in meshes]
    ds.set_vertices(np.concatenate(moved))
    ds.refit(kd.REFIT_VERTICES)
    for i in sorted(set(range(min(len(sizes), 64))) | set(range(max(len(sizes) - 65, 0), len(sizes)))):
        vol, tet = ds.read_tree(i)
        if not sizes[i]:
            assert len(tet) == 0
            continue
        want_vol, want_tet = preorder(oracle.leaf_dops(K, moved[i], meshes[i].tets), tet[tet >= 0])
        assert np.array_equal(tet, want_tet) and np.array_equal(vol, want_vol), (i, sizes[i])
    # the roots as the traversal sees them
    if len(sizes) > 1:
        pairs = np.stack([np.arange(len(sizes)), np.roll(np.arange(len(sizes)), 1)], 1).astype(np.uint32)
        ds.traverse_sync(pairs)
        want = [np.zeros((0, 3), np.int64)]
        for p, (a, b) in enumerate(pairs[:12]):
            if sizes[a] and sizes[b]:
                rows, _, _ = oracle.run_pair(K, moved[a], meshes[a].tets, meshes[a].surf, moved[b], meshes[b].tets,
                                             meshes[b].surf, restA=meshes[a].xyz, restB=meshes[b].xyz)
                want.append(np.column_stack([np.full(len(rows), p), rows]))
        got = ds.candidates()
        got = got[got[:, 0] < 12].astype(np.int64)
        want = np.concatenate(want).astype(np.int64)
        assert np.array_equal(got[np.lexsort(got.T[::-1])], want[np.lexsort(want.T[::-1])])
    ds.close()
