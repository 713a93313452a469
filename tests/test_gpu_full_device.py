"""A broad phase that finds no device memory for its pairs reports it, and the next
queries work."""
import contextlib
import ctypes

import numpy as np
import pytest

import kdop_b200 as kd
from kdop_b200 import scenes

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def full_device():
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
        yield
    finally:
        for d in taken:
            rt.cudaFree(d)


def test_broad_phase_without_room(ctx):
    n = 700
    ds = kd.DeviceScene(ctx, 6, [scenes.lattice(1)] * n)
    rng = np.random.default_rng(0)
    far = rng.uniform(-20, 20, (n, 3)).astype(np.float32)
    few = ds.broad_phase(far)
    near = (far * np.float32(1e-3)).astype(np.float32)
    every = np.stack(np.triu_indices(n, 1), 1)
    assert 0 < len(few) < 20000 and 10 * len(every) > (2 << 20)
    held = ds.info()["device_bytes"]
    with full_device():
        for _ in range(2):
            with pytest.raises(kd.KdopError):
                ds.broad_phase(near)
    assert ds.info()["device_bytes"] <= held
    assert np.array_equal(ds.broad_phase(far), few)
    assert np.array_equal(ds.broad_phase(near), every)
    assert np.array_equal(ds.broad_phase(far), few)
    ds.close()
