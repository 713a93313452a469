"""The counters a call reads back are those of the work enqueued last: across
repeated calls, graph steps, another set of contacts, and replays of a graph the
caller captured (work that runs without a call of the library)."""
import numpy as np
import pytest

import kdop_b200 as kd
from kdop_b200 import scenes

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_counters_follow_what_was_enqueued(ctx):
    sc = scenes.config5(n_pairs=3, n=5)
    ds = kd.DeviceScene(ctx, sc.K, sc.meshes)
    far = sc.pos.copy()
    far[1::2] += 100.0
    counts = {}
    for name, pos in (("near", sc.pos), ("far", far)):
        ds.set_poses(sc.quat, pos)
        ds.refit(kd.REFIT_POSE)
        st = ds.traverse_sync(sc.pairs, contacts=True)
        counts[name] = (st.n_tests, st.n_candidates, st.n_contacts)
        assert ds.stats().n_tests == st.n_tests and len(ds.candidates()) == st.n_candidates
        assert len(ds.read_contacts()) == st.n_contacts
    assert counts["near"][2] > 0 and counts["far"][2] == 0
    ds.graph_capture(sc.pairs)
    for name, pos in (("near", sc.pos), ("far", far), ("near", sc.pos)):
        ds.set_poses(sc.quat, pos)
        ds.graph_launch()
        st = ds.stats()
        assert (st.n_tests, st.n_candidates, st.n_contacts) == counts[name]
        ds.sort_results()
        assert len(ds.read_contacts()) == counts[name][2] and ds.stats().n_contacts == counts[name][2]
    # contacts again, from other vertices, over the same candidates
    ds.set_poses(sc.quat, far)
    ds.refit(kd.REFIT_POSE)
    ds.contacts()
    assert ds.stats().n_contacts == 0 and ds.stats().n_candidates == counts["near"][1]


def test_counters_after_replays_of_a_captured_graph():
    stream = torch.cuda.Stream()
    ctx = kd.Context(0, stream=stream.cuda_stream)
    sc = scenes.config5(n_pairs=2, n=5)
    ds = kd.DeviceScene(ctx, sc.K, sc.meshes)
    ds.set_poses(sc.quat, sc.pos)
    ds.refit(kd.REFIT_POSE)
    near = torch.from_numpy(ds.read_vertices()).cuda()
    ds.set_vertices(near)
    ds.refit(kd.REFIT_VERTICES)
    n = ds.traverse_sync(sc.pairs, contacts=True).n_contacts
    x = near.clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="relaxed"):
        ds.set_vertices(x)
        ds.refit(kd.REFIT_VERTICES)
        ds.contacts()
    first = int(ds.v_off[1])
    for shift, want in ((0.0, n), (50.0, 0), (0.0, n)):
        with torch.cuda.stream(stream):
            x.copy_(near)
            x[first:int(ds.v_off[2])] += shift
            x[int(ds.v_off[3]):] += shift
            graph.replay()
        assert ds.stats().n_contacts == want and len(ds.read_contacts()) == want
    assert n > 0
    del graph
