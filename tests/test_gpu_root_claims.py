"""Claims of several root pairs or frontier entries at once (init_chunk): the
same tests and candidates on every route, entries of many pairs in one deque,
and a queue that is used about as much as with single claims -- waiting warps
are given claimed entries, not ever smaller parts of the first one."""
import ctypes as C

import numpy as np
import pytest
import torch

import kdop_b200 as kd
from kdop_b200 import scenes
from conftest import sorted_rows

pytestmark = pytest.mark.gpu


def posed(ctx, sc):
    ds = kd.DeviceScene(ctx, sc.K, sc.meshes)
    ds.set_poses(sc.quat, sc.pos)
    ds.refit(kd.REFIT_POSE)
    return ds


@pytest.mark.parametrize("load_group", [1, 2, 4, 8])
@pytest.mark.parametrize("chunk", [2, 31, 32])
@pytest.mark.parametrize("K", [6, 26])
def test_routes_agree(ctx, K, chunk, load_group):
    sc = scenes.small_batch(n_pairs=70, n_lo=1, n_hi=5, seed=9, K=K)
    ds = posed(ctx, sc)
    # pairs that end at the root among the others
    pairs = np.concatenate([sc.pairs, np.stack([sc.pairs[:, 0], np.roll(sc.pairs[:, 1], 1)], 1)])
    st = ds.traverse_sync(pairs)
    want = sorted_rows(ds.candidates())
    for kw in ({"wave_pairs": len(pairs)}, {"wave_pairs": 33}, {"mode": kd.TRAVERSE_PLAIN}, {}):
        # the smallest deques, eager donation: claimed entries are given away too
        o = ds.opts(init_chunk=chunk, load_group=load_group, stack_cap=64, donate_min=2, **kw)
        got = ds.traverse_sync(pairs, o)
        assert got.n_tests == st.n_tests and np.array_equal(sorted_rows(ds.candidates()), want), kw
    tests, rows = 0, []
    for rank in range(3):
        ds.traverse_shard(pairs, rank, 3, 64, ds.opts(init_chunk=chunk, load_group=load_group))
        tests += ds.stats().n_tests
        rows.append(ds.candidates())
    assert tests == st.n_tests and np.array_equal(sorted_rows(np.concatenate(rows)), want)


@pytest.mark.parametrize("chunk", [4, 32])
def test_queue_use(ctx, chunk):
    sc = scenes.config3(32, 5, 1000, 6000, 0.15, 14)
    ds = posed(ctx, sc)
    ds.traverse_sync(sc.pairs)
    ds.reserve(queue=1 << 22)

    def used(c):
        o = ds.opts(init_chunk=c, wave_pairs=32)
        out = []
        for _ in range(5):
            ds.traverse(sc.pairs, o)
            out.append(ds.stats().queue_used)
        return max(out)

    assert used(chunk) <= 1.5 * used(1)


@pytest.mark.parametrize("chunk", [1, 4, 32])
def test_traversal_without_allocation(ctx, chunk):
    # 64 touching pairs: 23,000 to 29,000 of the static queue's 65,536 entries
    sc = scenes.config5(64, 10, 3, 14)
    ds = posed(ctx, sc)
    st = ds.traverse_sync(sc.pairs)
    pairs = torch.from_numpy(sc.pairs.view(np.int32)).cuda()
    cap = int(st.n_candidates) + 64
    cand = torch.zeros(3 * cap, dtype=torch.int32, device="cuda")
    counters = torch.zeros(4, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    o = ds.opts(init_chunk=chunk)
    fn = ds.lib.kdop_traverse_noalloc
    fn.argtypes = [C.c_void_p, C.c_int64, C.c_void_p, C.c_void_p, C.c_int64, C.c_void_p, C.c_void_p]
    assert fn(ds.h, 64, pairs.data_ptr(), cand.data_ptr(), cap, counters.data_ptr(), C.byref(o)) == 0
    ctx.synchronize()
    assert counters.tolist() == [st.n_candidates, st.n_tests, st.n_leaf_overlaps, 0]
