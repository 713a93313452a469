"""Root pairs are taken by decreasing size, equal sizes in list order, whether the
host or the device orders them: in waves of one pair the rows appear in that order."""
import numpy as np
import pytest

import kdop_b200 as kd
from kdop_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_pairs", [1, 2, 256, 257, 1025, 8192, 8193])
def test_largest_pairs_first(ctx, n_pairs):
    rng = np.random.default_rng(n_pairs)
    whole = [scenes.lattice(1, 0.1, rng) for _ in range(30)]
    tets = rng.integers(1, 7, len(whole))
    meshes = [scenes.Mesh(m.xyz, m.tets[:k], m.surf[:k]) for m, k in zip(whole, tets)]
    meshes[4] = scenes.Mesh(np.zeros((0, 3), np.float32), np.zeros((0, 4), np.uint32), np.zeros(0, np.uint8))
    tets[4] = 0
    ds = kd.DeviceScene(ctx, 14, meshes)
    pairs = rng.integers(0, len(meshes), (n_pairs, 2)).astype(np.uint32)
    if n_pairs <= 2:
        pairs = np.array([[0, 1], [2, 3]], np.uint32)[:n_pairs]
    order = np.argsort(-(tets[pairs[:, 0]] + tets[pairs[:, 1]]), kind="stable")
    ds.traverse_sync(pairs, ds.opts(wave_pairs=1, surface_filter=0))
    rows = ds.candidates()[:, 0]
    got = rows[np.concatenate([[True], rows[1:] != rows[:-1]])]
    assert len(set(got)) == len(got)  # a pair's rows are together
    assert np.array_equal(got, order[np.isin(order, got)])
    assert len(got) > 0.5 * n_pairs
    ds.close()
