"""Steps whose lists grow a little each time take new device memory only now and
then, and give what a scene made for the last list gives."""
import numpy as np
import pytest

import kdop_b200 as kd
from conftest import sorted_rows
from kdop_b200 import scenes

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bodies, first, steps", [(2, 1, 40), (20, 20, 100), (40, 250, 40)])
def test_pair_list_grows_by_one(ctx, bodies, first, steps):
    sc = scenes.config5(n_pairs=bodies // 2, n=3)
    rng = np.random.default_rng(bodies)
    pairs = rng.integers(0, bodies, (first + steps, 2)).astype(np.uint32)
    ds = kd.DeviceScene(ctx, sc.K, sc.meshes)
    ds.set_poses(sc.quat, sc.pos)
    ds.refit(kd.REFIT_POSE)
    ds.traverse_sync(pairs[:first])
    held = set()
    for n in range(first + 1, first + steps + 1):
        st = ds.traverse_sync(pairs[:n])
        held.add(ds.info()["device_bytes"])
    # a block holds a quarter and 16 pairs more than the list it was made for
    assert len(held) <= 6
    other = kd.DeviceScene(ctx, sc.K, sc.meshes)
    other.set_poses(sc.quat, sc.pos)
    other.refit(kd.REFIT_POSE)
    assert other.traverse_sync(pairs).n_tests == st.n_tests
    assert np.array_equal(sorted_rows(ds.candidates()), sorted_rows(other.candidates()))
    ds.close()
    other.close()


@pytest.mark.parametrize("n_pairs", [21, 200, 300])
def test_longer_list_inside_a_callers_capture(n_pairs):
    stream = torch.cuda.Stream()
    ctx = kd.Context(0, stream=stream.cuda_stream)
    sc = scenes.config5(n_pairs=10, n=3)
    rng = np.random.default_rng(n_pairs)
    pairs = rng.integers(0, 20, (n_pairs, 2)).astype(np.uint32)
    ds = kd.DeviceScene(ctx, sc.K, sc.meshes)
    ds.set_poses(sc.quat, sc.pos)
    ds.refit(kd.REFIT_POSE)
    ds.traverse_sync(pairs[:20])
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="relaxed"):
        ds.traverse(pairs)
    ds.candidates()  # of the traversal before, the list already the next one's: any rows, no fault
    with torch.cuda.stream(stream):
        graph.replay()
    other = kd.DeviceScene(ctx, sc.K, sc.meshes)
    other.set_poses(sc.quat, sc.pos)
    other.refit(kd.REFIT_POSE)
    assert ds.stats().n_tests == other.traverse_sync(pairs).n_tests
    assert np.array_equal(sorted_rows(ds.candidates()), sorted_rows(other.candidates()))
    del graph


@pytest.mark.parametrize("n_pairs, between", [(300, 10), (40, 400), (40, 250), (1, 256)])
def test_replay_of_a_list_after_another(n_pairs, between):
    """The results are those of the graph's list, whatever list a call had in between."""
    stream = torch.cuda.Stream()
    ctx = kd.Context(0, stream=stream.cuda_stream)
    sc = scenes.config5(n_pairs=10, n=3)
    rng = np.random.default_rng(n_pairs)
    pairs = rng.integers(0, 20, (n_pairs, 2)).astype(np.uint32)
    ds = kd.DeviceScene(ctx, sc.K, sc.meshes)
    ds.set_poses(sc.quat, sc.pos)
    ds.refit(kd.REFIT_POSE)
    ds.traverse_sync(rng.integers(0, 20, (max(n_pairs, between), 2)).astype(np.uint32))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="relaxed"):
        ds.traverse(pairs)
        ds.contacts()
    ds.traverse_sync(rng.integers(0, 20, (between, 2)).astype(np.uint32), contacts=True)
    with torch.cuda.stream(stream):
        graph.replay()
    other = kd.DeviceScene(ctx, sc.K, sc.meshes)
    other.set_poses(sc.quat, sc.pos)
    other.refit(kd.REFIT_POSE)
    other.traverse_sync(pairs, contacts=True)
    for scene in (ds, other):
        scene.sort_results()
    assert np.array_equal(ds.candidates(), other.candidates())
    assert ds.read_contacts().tobytes() == other.read_contacts().tobytes()
    for got, want in zip(ds.reduce_contacts(), other.reduce_contacts()):
        assert got.tobytes() == want.tobytes()
    del graph


def test_candidates_grow_from_step_to_step(ctx):
    sc = scenes.touching_pair(n=8, seed=0, K=14)
    ds = kd.DeviceScene(ctx, sc.K, sc.meshes)
    axis = sc.pos[1] - sc.pos[0]
    held, counts = set(), []
    for k in range(60):
        pos = sc.pos.copy()
        pos[1] -= np.float32(0.01 * k) * axis
        ds.set_poses(sc.quat, pos)
        ds.refit(kd.REFIT_POSE)
        ds.traverse_sync(sc.pairs)
        counts.append(len(ds.candidates()))
        held.add(ds.info()["device_bytes"])
    assert counts[-1] > 2 * counts[0] and len(set(counts)) > 30
    # a quarter more room each time it runs out
    assert len(held) <= 3 + np.log(max(counts) / min(counts)) / np.log(1.25)
    ds.close()
