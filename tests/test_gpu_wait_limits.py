"""Waits of the sorts and one-pass scans that run out (the test hook leaves the
first tile without a block): the call reports KDOP_ERR_TIMEOUT, nothing reads
the incomplete order, lost results are refused, and the context goes on."""
import numpy as np
import pytest

import kdop_b200 as kd
from kdop_b200 import scenes
from conftest import sorted_rows

pytestmark = pytest.mark.gpu

TIMEOUT, STATE = kd.lib.ERR_TIMEOUT, kd.lib.ERR_STATE
LIMIT = 20  # ms
SORT, SCAN = 1, 2


@pytest.fixture
def own(cuda_library_path):
    c = kd.Context(0)
    yield c
    c.set_wait_limit()


def status(fn):
    with pytest.raises(kd.KdopError) as e:
        fn()
    return e.value.status


@pytest.mark.parametrize("stuck", [SORT, SCAN, SORT + SCAN])
@pytest.mark.parametrize("n,bodies,ties", [(8193, 4, False), (50000, 1 << 20, False), (50000, 2, True)])
def test_reduction(own, stuck, n, bodies, ties):
    rng = np.random.default_rng(n)
    rows = np.zeros(n, kd.CONTACT_DTYPE)
    rows["p"] = rng.uniform(-1, 1, (n, 3))
    if ties:
        rows["p"][:, 1] = 0.5  # one run of p.y: the long runs' sorts as well
    rows["cand"] = np.arange(n)
    pair = rng.integers(0, bodies, (n, 2)).astype(np.uint32)
    want, want_bodies = own.reduce_contact_rows(rows, pair)
    own.set_wait_limit(LIMIT, stuck)
    assert status(lambda: own.reduce_contact_rows(rows, pair)) == TIMEOUT
    own.set_wait_limit()
    got, got_bodies = own.reduce_contact_rows(rows, pair)
    assert got.tobytes() == want.tobytes() and np.array_equal(got_bodies, want_bodies)


@pytest.mark.parametrize("stuck", [SORT, SCAN])
@pytest.mark.parametrize("two_sorts", [False, True])
def test_results(own, stuck, two_sorts):
    sc = scenes.config5(8, 10, 7, 14)
    ds = kd.DeviceScene(own, sc.K, sc.meshes)
    ds.set_poses(sc.quat, sc.pos)
    ds.refit(kd.REFIT_POSE)

    def step():
        st = ds.traverse_sync(sc.pairs, contacts=True)
        assert st.n_candidates > 8192 and st.n_contacts > 0
        if two_sorts:  # the scene's list is the captured step's now, not the results'
            ds.graph_capture(sc.pairs, kd.REFIT_POSE)

    step()
    ds.sort_results()
    want, contacts = ds.candidates(), ds.read_contacts()
    step()
    own.set_wait_limit(LIMIT, stuck)
    assert status(ds.sort_results) == TIMEOUT
    own.set_wait_limit()
    grad = np.zeros((ds.v_off[-1], 3), np.float32)
    ones = np.ones(len(contacts), np.float32)
    for call in (ds.sort_results, ds.candidates, ds.contacts, ds.read_contacts, lambda: ds.adjoint(ones, None, grad)):
        assert status(call) == STATE
    assert status(ds.reduce_contacts) == STATE
    if two_sorts:
        ds.graph_launch()
    else:
        step()
    ds.sort_results()
    assert np.array_equal(ds.candidates(), want)
    assert ds.read_contacts().tobytes() == contacts.tobytes()


def test_tree_build(own):
    mesh = scenes.lattice(16, 0.1, np.random.default_rng(1))
    want = kd.DeviceScene(own, 14, [mesh] * 2).read_tree(1)
    own.set_wait_limit(LIMIT, SORT)
    assert status(lambda: kd.DeviceScene(own, 14, [mesh] * 2)) == TIMEOUT
    own.set_wait_limit()
    got = kd.DeviceScene(own, 14, [mesh] * 2).read_tree(1)
    assert all(np.array_equal(a, b) for a, b in zip(got, want))


def test_broad_phase(own):
    rng = np.random.default_rng(2)
    ds = kd.DeviceScene(own, 6, [scenes.lattice(1, 0.1, rng)] * 100)
    pos = rng.uniform(-3, 3, (100, 3)).astype(np.float32)
    want = ds.broad_phase(pos)
    own.set_wait_limit(LIMIT, SCAN)
    assert status(lambda: ds.broad_phase(pos)) == TIMEOUT
    own.set_wait_limit()
    assert len(want) and np.array_equal(ds.broad_phase(pos), want)


@pytest.mark.parametrize("shard", [False, True])
def test_traversal_orders(own, shard):
    # the root pairs' order (16,000 pairs), and a shard's frontier (16,384 node pairs at least)
    sc = scenes.config3(24, 5, 4000, 6000, 0.3, 14) if shard else scenes.config5(8, 10, 7, 14)
    ds = kd.DeviceScene(own, sc.K, sc.meshes)
    ds.set_poses(sc.quat, sc.pos)
    ds.refit(kd.REFIT_POSE)
    pairs = sc.pairs if shard else np.tile(sc.pairs, (2000, 1))
    ds.traverse_sync(pairs)

    def go(**kw):
        if shard:
            ds.traverse_shard(pairs, 0, 1, 16384, ds.opts(**kw))
        else:
            ds.traverse(pairs, ds.opts(**kw))
        return ds.stats(check=False)

    st = go()
    assert st.status == 0 and st.n_candidates > 0
    want = sorted_rows(ds.candidates()) if shard else None
    own.set_wait_limit(0, SORT)
    assert go(timeout_ms=LIMIT).status == TIMEOUT
    own.set_wait_limit()
    again = go()
    assert (again.status, again.n_tests, again.n_candidates) == (0, st.n_tests, st.n_candidates)
    if shard:
        assert np.array_equal(sorted_rows(ds.candidates()), want)
