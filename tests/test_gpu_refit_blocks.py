"""The refit's blocks at the tet counts where their shape changes: trees of one
node, of less than a warp, of a warp and of a block, one more and one less, and
trees refitted in two and three launches; odd numbers of trees (a padding
root), empty meshes, host-built trees and given leaf orders.  Every node's
slabs equal the oracle's bit for bit, after poses and after new vertices."""
import numpy as np
import pytest

import kdop_b200 as kd
from kdop_b200 import scenes

pytestmark = pytest.mark.gpu

COUNTS = [1, 2, 3, 4, 5, 31, 32, 33, 63, 64, 65, 127, 128, 255, 256, 257, 383, 511, 512, 513, 1023, 1024, 1537]


def soup(n, rng):
    """n tets of positive orientation over a jittered lattice's vertices."""
    m = scenes.lattice(max(1, int(np.ceil((n / 6) ** (1 / 3)))), 0.1, rng)
    pick = np.sort(rng.permutation(m.n_tets)[:n])
    tets = np.ascontiguousarray(m.tets[pick])
    return scenes.Mesh(m.xyz, tets, scenes.surface_map(tets))


def check(oracle, ds, mesh, i, K, world):
    """Leaves hold their tet's slabs, inner nodes the union of their children (preorder)."""
    vol, tet = ds.read_tree(i)
    n = mesh.n_tets
    assert len(vol) == max(2 * n - 1, 0)
    leaf = tet >= 0
    assert sorted(tet[leaf]) == list(range(n))
    want = oracle.leaf_dops(K, world, mesh.tets)
    assert np.array_equal(vol[leaf].view(np.uint32), want[tet[leaf]].view(np.uint32))

    def walk(at, size):
        if size == 1:
            assert leaf[at]
            return vol[at]
        left = size - size // 2
        a, b = walk(at + 1, left), walk(at + 2 * left, size - left)
        u = np.empty(K, np.float32)
        u[0::2], u[1::2] = np.minimum(a[0::2], b[0::2]), np.maximum(a[1::2], b[1::2])
        assert not leaf[at] and np.array_equal(vol[at].view(np.uint32), u.view(np.uint32))
        return u

    if n:
        walk(0, n)


@pytest.mark.parametrize("K", scenes.SUPPORTED_K)
@pytest.mark.parametrize("build", [kd.BUILD_DEVICE, kd.BUILD_HOST])
def test_refit_equals_leaf_slabs_and_unions(ctx, oracle, K, build):
    rng = np.random.default_rng(K)
    counts = COUNTS if build == kd.BUILD_DEVICE else COUNTS[::3]
    meshes = [soup(n, rng) for n in counts]
    meshes.insert(3, scenes.Mesh(np.zeros((0, 3), np.float32), np.zeros((0, 4), np.uint32), np.zeros(0, np.uint8)))
    meshes[5].leaf_order = rng.permutation(meshes[5].n_tets).astype(np.uint32)
    if len([m for m in meshes if m.n_tets]) % 2 == 0:
        meshes.append(soup(7, rng))  # an odd number of roots
    n = len(meshes)
    quat = np.stack([scenes.random_quaternion(rng) for _ in range(n)])
    pos = rng.uniform(-5, 5, (n, 3)).astype(np.float32)
    ds = kd.DeviceScene(ctx, K, meshes, build=build)
    for mode in (kd.REFIT_POSE, kd.REFIT_VERTICES):
        if mode == kd.REFIT_POSE:
            ds.set_poses(quat, pos)
            worlds = [oracle.rotate(quat[i], pos[i], m.xyz) if m.n_verts else m.xyz for i, m in enumerate(meshes)]
        else:
            worlds = [(m.xyz + rng.uniform(-0.2, 0.2, m.xyz.shape)).astype(np.float32) for m in meshes]
            worlds[0][:, 1] = 0.0
            worlds[0] *= np.float32(-1)  # negative zeros
            ds.set_vertices(np.concatenate(worlds))
        ds.refit(mode)
        for i, m in enumerate(meshes):
            check(oracle, ds, m, i, K, worlds[i])


def test_refit_of_non_finite_vertices(ctx, oracle):
    rng = np.random.default_rng(2)
    mesh = soup(600, rng)
    world = mesh.xyz.copy()
    bad = rng.permutation(len(world))[:60]
    world[bad, rng.integers(0, 3, 60)] = rng.choice(np.array([np.inf, -np.inf, np.nan, 3.0e38, -3.0e38], np.float32), 60)
    for K in (14, 26):
        ds = kd.DeviceScene(ctx, K, [mesh])
        ds.set_vertices(world)
        ds.refit(kd.REFIT_VERTICES)
        check(oracle, ds, mesh, 0, K, world)


@pytest.mark.parametrize("n", [20, 23])
def test_refit_in_three_launches(ctx, oracle, n):
    rng = np.random.default_rng(n)
    mesh = scenes.lattice(n + 8, 0.2, rng)  # 131,712 and 178,746 tets: 18 levels
    ds = kd.DeviceScene(ctx, 18, [mesh, scenes.lattice(2, 0.1, rng)])
    assert mesh.n_tets > 1 << 16
    check(oracle, ds, mesh, 0, 18, mesh.xyz)


@pytest.mark.parametrize("K", [14, 18, 26])
def test_refit_of_a_large_forest(ctx, oracle, K):
    # above 2,048 blocks of 256 nodes the first launch's warps stop on their own
    rng = np.random.default_rng(K)
    big = scenes.lattice(46, 0.2, rng)  # 584,016 tets: 2^19 nodes of depth 19
    meshes = [soup(n, rng) for n in (1, 31, 32, 33, 64, 65, 130, 300, 5000)] + [big]
    meshes += [soup(2, rng)] * (1 - len(meshes) % 2)
    ds = kd.DeviceScene(ctx, K, meshes)
    worlds = [(m.xyz + rng.uniform(-0.1, 0.1, m.xyz.shape)).astype(np.float32) for m in meshes]
    ds.set_vertices(np.concatenate(worlds))
    ds.refit(kd.REFIT_VERTICES)
    for i, m in enumerate(meshes):
        if m is not big:
            check(oracle, ds, m, i, K, worlds[i])
            continue
        vol, tet = ds.read_tree(i)
        leaf = tet >= 0
        assert np.array_equal(np.sort(tet[leaf]), np.arange(m.n_tets))
        assert np.array_equal(vol[leaf], oracle.leaf_dops(K, worlds[i], m.tets)[tet[leaf]])
        at, size = np.array([0]), np.array([m.n_tets])
        while len(at):  # a level's nodes against their children
            at, size = at[size > 1], size[size > 1]
            left = size - size // 2
            a, b = at + 1, at + 2 * left
            assert not leaf[at].any()
            assert np.array_equal(vol[at, 0::2], np.minimum(vol[a, 0::2], vol[b, 0::2]))
            assert np.array_equal(vol[at, 1::2], np.maximum(vol[a, 1::2], vol[b, 1::2]))
            at = np.stack([a, b], 1).ravel()
            size = np.stack([left, size - left], 1).ravel()
