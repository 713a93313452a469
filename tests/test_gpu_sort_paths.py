"""The device radix sort, its one-pass scans and the reduction built on them at
the sizes where their path changes: one block, tiles and their remainders,
small and large tiles, keys of one and of two sorts, runs ranked row by row and
runs sorted on their own.  Exact against the oracle's restatement."""
import numpy as np
import pytest

import kdop_b200 as kd
from kdop_b200 import scenes
from conftest import sorted_rows

pytestmark = pytest.mark.gpu


def contacts(rows7):
    c = np.zeros(len(rows7), kd.CONTACT_DTYPE)
    c["p"], c["n"], c["depth"] = rows7[:, 0:3], rows7[:, 3:6], rows7[:, 6]
    c["cand"] = np.arange(len(rows7))
    return c


def check(ctx, oracle, rows, bodies):
    want_r, want_b, want_src = oracle.reduce_contacts(rows, bodies)
    out, ob = ctx.reduce_contact_rows(contacts(rows), bodies)
    assert np.array_equal(ob, want_b)
    assert np.array_equal(out["cand"], want_src)
    assert np.all(np.column_stack([out["p"], out["n"], out["depth"][:, None]]) == want_r)


@pytest.mark.parametrize("n", [1, 2, 1023, 1024, 1025, 2049, 4095, 4096, 4097, 6144, 8191, 70001])
@pytest.mark.parametrize("body_max", [0, 3, 70000, 2 ** 32 - 1])
def test_reduction_sizes_and_body_widths(ctx, oracle, n, body_max):
    rng = np.random.default_rng(n + body_max % 97)
    # few distinct values a field: runs and ties at every level of the order
    rows = (rng.integers(0, 12, (n, 7)) * np.float32(0.25) - np.float32(1.0)).astype(np.float32)
    rows[rng.random((n, 7)) < 0.05] *= -1  # signed zeros among them
    rows[:, 0] += rng.integers(0, 3, n) * np.float32(5e-7)  # near duplicates within the tolerance
    bodies = rng.choice(np.unique(np.array([0, body_max // 3, body_max], np.uint64)), (n, 2)).astype(np.uint32)
    check(ctx, oracle, rows, bodies)


@pytest.mark.parametrize("run", [511, 512, 513, 5000])
def test_long_runs(ctx, oracle, run):
    # two runs of equal p.y (one side and the other of the row-by-row limit) among rows of their own
    rng = np.random.default_rng(run)
    rows = rng.uniform(-2, 2, (run + 512 + 3000, 7)).astype(np.float32)
    rows[:run, 1] = np.float32(0.5)
    rows[run:run + 512, 1] = np.float32(-0.25)
    rows[:run // 2, 0] = np.float32(1.0)  # half of the run also shares p.x
    rows[run // 4:run // 3] = rows[:run // 3 - run // 4]  # and some rows are equal
    rows = rows[rng.permutation(len(rows))]
    check(ctx, oracle, rows, np.zeros((len(rows), 2), np.uint32))


@pytest.mark.parametrize("n_pairs,lo,hi", [(1, 2, 2), (3, 3, 6), (40, 2, 9)])
def test_result_order_with_and_without_the_pair_list(ctx, n_pairs, lo, hi):
    # a capture replaces the scene's pair list, so the results made before it are ordered without it
    sc = scenes.small_batch(n_pairs=n_pairs, n_lo=lo, n_hi=hi, seed=5)
    ds = kd.DeviceScene(ctx, sc.K, sc.meshes)
    ds.set_poses(sc.quat, sc.pos)
    ds.refit(kd.REFIT_POSE)
    ds.reserve(candidates=1 << 20, contacts=1 << 20)
    got = []
    for capture in (False, True):
        ds.traverse_sync(sc.pairs, contacts=True)
        want = sorted_rows(ds.candidates())
        if capture:
            ds.graph_capture(sc.pairs)
        ds.sort_results()
        assert np.array_equal(ds.candidates(), want)
        got.append(ds.read_contacts().copy())
    assert len(got[0]) == len(got[1]) and np.array_equal(got[0].view(np.uint8), got[1].view(np.uint8))
