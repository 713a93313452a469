"""Rows and nodes on their way out are staged apart from host arrays on their
way in: a read-back leaves the buffer of an upload that a caller captured where
it is, and takes smaller windows where the device has no room for one."""
import ctypes

import numpy as np
import pytest

import kdop_b200 as kd
from conftest import sorted_rows
from kdop_b200 import scenes

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_captured_upload_after_read_backs():
    stream = torch.cuda.Stream()
    ctx = kd.Context(0, stream=stream.cuda_stream)
    sc = scenes.config5(n_pairs=2, n=5)
    ds = kd.DeviceScene(ctx, sc.K, sc.meshes)
    quat = torch.from_numpy(np.ascontiguousarray(sc.quat, np.float32)).pin_memory()
    pos = torch.from_numpy(np.ascontiguousarray(sc.pos, np.float32)).pin_memory()
    near = pos.clone()
    q, p = quat.numpy(), pos.numpy()
    ds.set_poses(q, p)
    ds.refit(kd.REFIT_POSE)
    n = ds.traverse_sync(sc.pairs, contacts=True).n_contacts
    assert n > 0
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="relaxed"):
        ds.set_poses(q, p)
        ds.refit(kd.REFIT_POSE)
        ds.contacts()
    # more words than the poses take, rows and trees
    assert 3 * len(ds.candidates()) > 7 * len(p)
    ds.read_tree(0)
    for shift, want in ((0.0, n), (50.0, 0), (0.0, n)):
        pos.copy_(near)
        p[1::2] += np.float32(shift)
        with torch.cuda.stream(stream):
            graph.replay()
        assert ds.stats().n_contacts == want
        assert len(ds.candidates()) > 0
    del graph


def test_read_backs_on_a_full_device(ctx):
    sc = scenes.config5(n_pairs=64, n=20)
    ds = kd.DeviceScene(ctx, sc.K, sc.meshes)
    ds.set_poses(sc.quat, sc.pos)
    ds.refit(kd.REFIT_POSE)
    st = ds.traverse_sync(sc.pairs)
    assert 12 * st.n_candidates > (2 << 20)
    # what the read-backs give with room, from a scene of its own
    other = kd.DeviceScene(ctx, sc.K, sc.meshes)
    other.set_poses(sc.quat, sc.pos)
    other.refit(kd.REFIT_POSE)
    other.traverse_sync(sc.pairs)
    rows, (vol, tet) = other.candidates(), other.read_tree(0)
    other.close()
    rt = ctypes.CDLL("libcudart.so.12")
    rt.cudaMalloc.argtypes = [ctypes.POINTER(ctypes.c_void_p), ctypes.c_size_t]
    rt.cudaFree.argtypes = [ctypes.c_void_p]
    torch.cuda.synchronize()
    taken = []
    try:
        for size in (1 << 30, 64 << 20, 2 << 20):
            while True:
                d = ctypes.c_void_p()
                if rt.cudaMalloc(ctypes.byref(d), size) != 0:
                    rt.cudaGetLastError()
                    break
                taken.append(d)
        rt.cudaFree(taken.pop())  # room for one block of 2 MB
        got, (vol2, tet2) = ds.candidates(), ds.read_tree(0)
    finally:
        for d in taken:
            rt.cudaFree(d)
    assert np.array_equal(sorted_rows(got), sorted_rows(rows))
    assert np.array_equal(vol2, vol) and np.array_equal(tet2, tet)
    ds.close()


def preorder(slabs, tets):
    """The tree over leaves `tets` in order, split at the index median, in preorder."""
    vol, tet = [], []

    def walk(f, n):
        at = len(vol)
        vol.append(None)
        tet.append(int(tets[f]) if n == 1 else -1)
        if n == 1:
            vol[at] = slabs[tets[f]]
            return vol[at]
        left = n - n // 2
        a, b = walk(f, left), walk(f + left, n - left)
        vol[at] = np.where(np.arange(slabs.shape[1]) % 2, np.maximum(a, b), np.minimum(a, b))
        return vol[at]

    walk(0, len(tets))
    return np.array(vol), np.array(tet)


# a node takes 4 K + 8 bytes: trees around the 64 KB that are read through pinned memory
@pytest.mark.parametrize("K,n_tets", [(6, 1), (6, 2), (6, 512), (14, 7), (14, 512), (14, 513), (26, 292), (26, 293)])
def test_small_trees(ctx, oracle, K, n_tets):
    rng = np.random.default_rng(n_tets)
    whole = scenes.lattice(5, 0.1, rng)
    mesh = scenes.Mesh(whole.xyz, whole.tets[:n_tets], whole.surf[:n_tets])
    ds = kd.DeviceScene(ctx, K, [scenes.lattice(1), mesh, whole])
    for m in (mesh, whole, mesh):  # the buffer of one read is another's
        vol, tet = ds.read_tree(1 if m is mesh else 2)
        want_vol, want_tet = preorder(oracle.leaf_dops(K, m.xyz, m.tets), tet[tet >= 0])
        assert np.array_equal(np.sort(tet[tet >= 0]), np.arange(m.n_tets))
        assert np.array_equal(tet, want_tet) and np.array_equal(vol, want_vol)
    ds.close()
