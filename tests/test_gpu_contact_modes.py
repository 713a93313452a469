"""Contact generation around the list lengths where its passes change from a
warp to a thread per candidate: copies of one mesh pair in a list give each
copy the same rows, bit for bit, in either form, and they equal the oracle's --
on ordinary, on exactly aligned (tied distances, coincident points) and on
non-finite geometry (forms compared with each other)."""
import numpy as np
import pytest

import kdop_b200 as kd
from kdop_b200 import scenes

pytestmark = pytest.mark.gpu


def geometry(kind, n=8):
    rng = np.random.default_rng(5)
    a, b = scenes.lattice(n, 0.15 if kind != "aligned" else 0.0, rng), scenes.lattice(n)
    xa, xb = a.xyz.copy(), b.xyz.copy()
    xb[:, 0] += np.float32(n - (0.25 if kind == "aligned" else 0.3))
    if kind == "bad":
        face = np.nonzero(xa[:, 0] > n / 2 - 0.5)[0]
        pick = rng.permutation(face)[:8]
        xa[pick, rng.integers(0, 3, 8)] = rng.choice(np.array([np.nan, np.inf, -np.inf, 2e38], np.float32), 8)
    return a, b, xa, xb


def copies(ctx, a, b, world, n):
    ds = kd.DeviceScene(ctx, 14, [a, b])
    ds.set_vertices(world)
    ds.refit(kd.REFIT_VERTICES)
    ds.traverse_sync(np.tile(np.array([[0, 1]], np.uint32), (n, 1)), contacts=True)
    ds.sort_results()
    cand, rows = ds.candidates(), ds.read_contacts()
    pair = cand[rows["cand"], 0]
    bits = np.column_stack([rows["p"].view(np.uint32), rows["n"].view(np.uint32), rows["depth"].view(np.uint32)])
    return cand, [bits[pair == k] for k in range(n)], rows


@pytest.mark.parametrize("kind", ["jittered", "aligned", "bad"])
def test_copies_agree_across_list_lengths(ctx, oracle, kind):
    a, b, xa, xb = geometry(kind)
    world = np.concatenate([xa, xb])
    cand, one, rows = copies(ctx, a, b, world, 1)
    per = len(cand)
    assert len(one[0]) > 100 and per < 4096
    if kind != "bad":
        want, _ = oracle.contacts(xa, a.tets, a.surf, xb, b.tets, b.surf, cand[:, 1:], "f")
        assert np.array_equal(np.asarray(want[:, :7], np.float32).view(np.uint32), one[0])
    lengths = sorted({2, 3, 4096 // per, 4096 // per + 1, 6144 // per, 6144 // per + 1, 8192 // per + 8,
                      24576 // per + 8})
    for n in lengths:
        _, many, _ = copies(ctx, a, b, world, n)
        for k in range(n):
            assert np.array_equal(many[k], one[0]), (n, k)
