"""Reduction of rows that tie: groups of one point within a run of equal p.y at the
sizes where ranking hands over to sorts, runs at theirs, duplicates, one or many
normals, and segments long enough for the walk's blocks of rows."""
import numpy as np
import pytest

import kdop_b200 as kd
from test_gpu_reduce import as_contacts, as_rows7

pytestmark = pytest.mark.gpu


def group(rng, run, tie, normals):
    """A run of `run` rows on one p.y, its points in groups of `tie`."""
    r = np.zeros((run, 7), np.float32)
    point = rng.uniform(-1, 1, (run, 2)).astype(np.float32)[np.arange(run) // tie]
    r[:, 0], r[:, 2] = point[:, 0], point[:, 1]
    r[:, 1] = np.float32(rng.uniform(-1, 1))
    r[:, 3:6] = rng.normal(size=(normals, 3)).astype(np.float32)[rng.integers(0, normals, run)]
    r[:, 6] = -rng.integers(0, 3, run).astype(np.float32) * np.float32(0.25)
    return r


@pytest.mark.parametrize("run,tie,normals", [(9, 9, 1), (100, 100, 1), (128, 128, 5), (129, 129, 5), (512, 127, 3),
                                             (512, 129, 3), (512, 512, 1), (512, 512, 500), (513, 1, 1), (513, 513, 40),
                                             (3000, 7, 2), (3000, 3000, 1)])
@pytest.mark.parametrize("runs", [1, 30])
def test_ties(ctx, oracle, run, tie, normals, runs):
    rng = np.random.default_rng(run * 7 + tie + runs)
    rows, bodies = [], []
    for k in range(runs):
        for length, t in ((run, tie), (int(rng.integers(1, 40)), 3)):
            rows.append(group(rng, length, t, normals))
            bodies.append(np.tile(np.uint32([k // 3, 50 + k % 3]), (length, 1)))
    rows, bodies = np.concatenate(rows), np.concatenate(bodies)
    p = rng.permutation(len(rows))
    rows, bodies = rows[p], bodies[p]
    want_r, want_b, want_src = oracle.reduce_contacts(rows, bodies)
    out, ob = ctx.reduce_contact_rows(as_contacts(rows), bodies)
    assert np.array_equal(ob, want_b)
    assert np.all(as_rows7(out) == want_r)
    assert np.array_equal(out["cand"], want_src)
