"""Pair lists at the lengths where their handling changes: the broad phase over
blocks of eight bodies and its remainders, with a list shorter than the answer,
and the root pairs' order made on the host and on the device."""
import ctypes as C

import numpy as np
import pytest

import kdop_b200 as kd
from kdop_b200 import scenes
from conftest import sorted_rows

pytestmark = pytest.mark.gpu


def bodies(n, seed):
    rng = np.random.default_rng(seed)
    pool = [scenes.lattice(k, 0.1, rng) for k in (1, 2, 3)]
    meshes = [pool[int(k)] for k in rng.integers(0, 3, n)]
    pos = rng.uniform(-1, 1, (n, 3)).astype(np.float32) * np.float32(1.5 * n ** (1 / 3))
    quat = np.stack([scenes.random_quaternion(rng) for _ in range(n)])
    return meshes, quat, pos


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 33, 64, 257, 1000])
def test_broad_phase_block_edges(ctx, oracle, n):
    meshes, quat, pos = bodies(n, n)
    ds = kd.DeviceScene(ctx, 6, meshes)
    ds.set_poses(quat, pos)
    want = oracle.broad_pairs(pos, np.array([oracle.mesh_radius(m.xyz) for m in meshes], np.float32))
    assert np.array_equal(ds.broad_phase(), want)
    assert np.array_equal(ds.broad_phase(pos), want)
    if len(want) > 1:
        short = np.zeros((len(want) - 1, 2), np.uint32)
        found = C.c_int64()
        rc = ds.lib.kdop_broad_phase(ds.h, None, kd.HOST, short.ctypes.data_as(C.c_void_p), len(short), C.byref(found))
        assert rc == kd.lib.ERR_CAPACITY and found.value == len(want) and not short.any()


@pytest.mark.parametrize("n_pairs", [255, 256, 257, 1024, 8193, 20000])
def test_pair_order_on_host_and_device(ctx, oracle, n_pairs):
    meshes, quat, pos = bodies(200, 3)
    meshes[4] = scenes.Mesh(np.zeros((0, 3), np.float32), np.zeros((0, 4), np.uint32), np.zeros(0, np.uint8))
    rng = np.random.default_rng(n_pairs)
    pairs = rng.integers(0, 200, (n_pairs, 2)).astype(np.uint32)
    ds = kd.DeviceScene(ctx, 14, meshes)
    ds.set_poses(quat, pos)
    ds.refit(kd.REFIT_POSE)
    st = ds.traverse_sync(pairs)
    got = sorted_rows(ds.candidates())
    roots = ds.traverse_sync(pairs, ds.opts(wave_pairs=n_pairs))
    assert st.n_tests == roots.n_tests and np.array_equal(got, sorted_rows(ds.candidates()))
    full = np.nonzero(~np.any(pairs == 4, axis=1))[0][:400]
    worlds = [oracle.rotate(quat[i], pos[i], m.xyz) if m.n_verts else m.xyz for i, m in enumerate(meshes)]
    order = [i for i in range(200) if i != 4]
    index = {m: k for k, m in enumerate(order)}
    sub = np.array([[index[int(a)], index[int(b)]] for a, b in pairs[full]], np.uint32)
    want, _, _ = oracle.run_pairs(14, [worlds[i] for i in order], [meshes[i] for i in order], sub)
    want[:, 0] = full[want[:, 0]]
    assert np.array_equal(got[np.isin(got[:, 0], full)], sorted_rows(want))
