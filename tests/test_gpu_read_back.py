"""Read-backs gathered on the device: a tree and a candidate list longer than
one staging window, trees behind others of every depth, repeated pairs."""
import numpy as np
import pytest

import kdop_b200 as kd
from kdop_b200 import scenes

pytestmark = pytest.mark.gpu


def test_tree_of_several_windows(ctx, oracle):
    # 471,858 tets, K = 26: 943,715 nodes of 28 words, two windows of 16 M words
    rng = np.random.default_rng(1)
    mesh = scenes.lattice(43, 0.2, rng)
    small = [scenes.lattice(n, 0.1, rng) for n in (1, 3, 5)]
    ds = kd.DeviceScene(ctx, 26, small + [mesh, small[0]])
    vol, tet = ds.read_tree(3)
    assert len(vol) * 28 > 16 << 20
    leaf = tet >= 0
    assert np.array_equal(np.sort(tet[leaf]), np.arange(mesh.n_tets))
    want = oracle.leaf_dops(26, mesh.xyz, mesh.tets)
    assert np.array_equal(vol[leaf], want[tet[leaf]])
    lo, hi = want[:, 0::2].min(axis=0), want[:, 1::2].max(axis=0)
    assert np.array_equal(vol[0, 0::2], lo) and np.array_equal(vol[0, 1::2], hi)


def test_candidates_of_several_windows(ctx):
    # every pair many times: more than 16 M / 3 rows, each copy the same list
    sc = scenes.config1()
    ds = kd.DeviceScene(ctx, sc.K, sc.meshes)
    ds.set_poses(sc.quat, sc.pos)
    ds.refit(kd.REFIT_POSE)
    opts = ds.opts(surface_filter=0)
    one = ds.traverse_sync(sc.pairs, opts).n_candidates
    want = ds.candidates()[:, 1:].astype(np.uint64)
    copies = int((16 << 20) // 3 // one + 2)
    ds.traverse_sync(np.repeat(sc.pairs, copies, axis=0), opts)
    ds.sort_results()
    rows = ds.candidates()
    assert len(rows) == copies * one > (16 << 20) // 3
    assert np.array_equal(rows[:, 0], np.repeat(np.arange(copies, dtype=np.uint32), one))
    key = np.sort((want[:, 0] << np.uint64(32)) | want[:, 1])
    got = ((rows[:, 1].astype(np.uint64) << np.uint64(32)) | rows[:, 2]).reshape(copies, one)
    assert np.array_equal(got, np.broadcast_to(key, got.shape))
