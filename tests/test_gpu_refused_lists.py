"""A pair list that is refused (a mesh index out of range) leaves the scene as
it was: results, their order, their reduction and the captured step still
belong to the list before it, however long the refused one is and wherever it
lies."""
import numpy as np
import pytest
import torch

import kdop_b200 as kd
from kdop_b200 import scenes

pytestmark = pytest.mark.gpu


def refused(sc, n, device):
    pairs = np.tile(sc.pairs, (n // len(sc.pairs) + 1, 1))[:n]
    pairs[n - 1, 1] = len(sc.meshes)
    return torch.from_numpy(pairs.view(np.int32)).cuda() if device else pairs


@pytest.mark.parametrize("device", [False, True])
@pytest.mark.parametrize("n", [1, 5, 257, 20000])
def test_results_of_the_list_before(ctx, n, device):
    sc = scenes.config5(5, 4, 7, 14)
    ds = kd.DeviceScene(ctx, sc.K, sc.meshes)
    ds.set_poses(sc.quat, sc.pos)
    ds.refit(kd.REFIT_POSE)
    st = ds.traverse_sync(sc.pairs, contacts=True)
    assert st.n_candidates > 0 and st.n_contacts > 0
    rows, (kept, bodies) = ds.candidates(), ds.reduce_contacts()
    with pytest.raises(kd.KdopError) as e:
        ds.traverse(refused(sc, n, device))
    assert e.value.status == kd.lib.ERR_INVALID
    assert np.array_equal(ds.candidates(), rows)
    again, again_bodies = ds.reduce_contacts()
    assert all(np.array_equal(again[f], kept[f]) for f in ("p", "n", "depth"))
    assert np.array_equal(again_bodies, bodies)
    ds.sort_results()
    assert np.array_equal(ds.candidates(), rows[np.lexsort(rows.T[::-1])])


@pytest.mark.parametrize("device", [False, True])
def test_captured_step_goes_on(ctx, device):
    sc = scenes.config5(5, 4, 7, 14)
    ds = kd.DeviceScene(ctx, sc.K, sc.meshes)
    ds.set_poses(sc.quat, sc.pos)
    ds.refit(kd.REFIT_POSE)
    st = ds.traverse_sync(sc.pairs, contacts=True)
    ds.sort_results()
    rows = ds.candidates()
    ds.graph_capture(sc.pairs, kd.REFIT_POSE)
    with pytest.raises(kd.KdopError):
        ds.traverse(refused(sc, 1000, device))
    ds.graph_launch()
    assert ds.stats().n_contacts == st.n_contacts
    ds.sort_results()
    assert np.array_equal(ds.candidates(), rows)


def test_results_survive_a_longer_list_that_follows(ctx):
    """The pairs of a longer accepted list replace the carried-over ones."""
    sc = scenes.config5(5, 4, 7, 14)
    ds = kd.DeviceScene(ctx, sc.K, sc.meshes)
    ds.set_poses(sc.quat, sc.pos)
    ds.refit(kd.REFIT_POSE)
    one = ds.traverse_sync(sc.pairs).n_candidates
    for n in (300, 9000):
        pairs = np.tile(sc.pairs[::-1], (n // 5, 1))
        ds.traverse_sync(pairs)
        ds.sort_results()
        rows = ds.candidates()
        assert len(rows) == one * (n // 5)
        first = rows[rows[:, 0] < 5]
        for k in range(n // 5):
            part = rows[rows[:, 0] // 5 == k].copy()
            part[:, 0] -= 5 * k
            assert np.array_equal(part, first)
            if k == 3:
                break
