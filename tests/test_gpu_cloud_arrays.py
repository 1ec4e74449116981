"""A cloud's arrays are cut from one slab and its stream comes from the idle ones: handles given other points again,
clouds created and destroyed on several threads, a caller's stream, and trimming between."""
import ctypes as C
import threading

import numpy as np
import pytest

from octrees_benchmark_b200.synth import lidar_tile

pytestmark = pytest.mark.gpu


def build(L, h, xyz):
    from octrees_benchmark_b200 import capi

    info = capi.OctTreeInfo()
    box = np.zeros(12)
    keys, perm = np.zeros(len(xyz), np.uint64), np.zeros(len(xyz), np.uint32)
    capi.check(L.oct_set_points(h, xyz.ctypes.data, len(xyz), 0), h)
    capi.check(L.oct_encode_sort(h, box.ctypes.data, keys.ctypes.data, perm.ctypes.data, None, 0), h)
    capi.check(L.oct_build(h, C.byref(info)), h)
    return keys, perm, info.n_total


def test_points_given_again(port):
    from octrees_benchmark_b200 import capi

    L, h = capi.lib(), C.c_void_p()
    capi.check(L.oct_cloud_create(C.byref(capi.OctParams(16, 5, 0, 0)), C.byref(h)), None)
    for n in (500, 40_000, 300, 40_000, 90_000, 0, 90_000, 1):
        xyz = lidar_tile(n, 60.0, seed=n) if n else np.zeros((0, 3))
        if n:
            keys, perm, total = build(L, h, xyz)
            k, p, box, _ = port.encode_sort(5, xyz)
            assert np.array_equal(keys, k) and np.array_equal(perm, p)
            assert total == port.build(5, k, 16, box).n_total
        else:
            build(L, h, xyz)
    capi.check(L.oct_cloud_destroy(h), None)


def test_threads_create_and_destroy():
    import torch

    from octrees_benchmark_b200 import LinearOctree, capi

    xyz = lidar_tile(8_000, 45.0, seed=2)
    want = LinearOctree(xyz).knn(xyz[:50], 5)
    bad = []

    def work(t):
        s = torch.cuda.Stream()
        for i in range(25):
            oc = LinearOctree(xyz, stream=s.cuda_stream if (i + t) % 3 == 0 else None)
            if not all(np.array_equal(a, b) for a, b in zip(want, oc.knn(xyz[:50], 5))):
                bad.append((t, i))
            oc.close()
            if i % 10 == 9:
                capi.lib().oct_trim_cloud_memory(0)

    ts = [threading.Thread(target=work, args=(t,)) for t in range(6)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not bad
