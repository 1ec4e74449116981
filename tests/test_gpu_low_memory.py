"""Calls that run out of device memory return an error, and the calls after them answer as before."""
import ctypes as C

import numpy as np
import pytest

from octrees_benchmark_b200.synth import lidar_tile

pytestmark = pytest.mark.gpu


@pytest.fixture
def scarce():
    """All of the device's memory but so many bytes, and the clouds' own pool, taken by the program."""
    import torch

    from octrees_benchmark_b200 import capi

    def take(left):
        capi.check(capi.lib().oct_trim_cloud_memory(0), None)
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        held.append(torch.empty(torch.cuda.mem_get_info()[0] - left, dtype=torch.uint8, device="cuda"))

    held = []
    yield take
    held.clear()
    torch.cuda.empty_cache()
    capi.check(capi.lib().oct_trim_cloud_memory(0), None)


def out_of_memory(call):
    from octrees_benchmark_b200 import capi

    with pytest.raises(capi.OctError) as e:
        call()
    assert e.value.status == capi.OCT_ERR_OUT_OF_MEMORY


def test_result_chunks_that_do_not_fit(scarce):
    from octrees_benchmark_b200 import LinearOctree

    xyz = lidar_tile(200_000, 140.0, seed=3)
    q = xyz[::10].copy()
    oc = LinearOctree(xyz, max_points_leaf=64)
    want = oc.radius_search(q, 2.0, "sphere"), oc.neighborsStruct(q, 2.0, "square"), oc.radius_hash(q, 2.0, "cube")
    scarce(3 << 30)
    out_of_memory(lambda: oc.radius_hash(q, 1e3, "sphere"))  # 4e9 results
    got = oc.radius_search(q, 2.0, "sphere"), oc.neighborsStruct(q, 2.0, "square"), oc.radius_hash(q, 2.0, "cube")
    for w, g in zip(want, got):
        assert all(np.array_equal(a, b) for a, b in zip(w, g))
    oc.close()


def test_points_that_do_not_fit_leave_the_cloud(scarce):
    from octrees_benchmark_b200 import LinearOctree, capi

    L = capi.lib()
    xyz = lidar_tile(50_000, 70.0, seed=4)
    q = xyz[::50].copy()
    oc = LinearOctree(xyz, max_points_leaf=64)
    want = [*oc.sorted_points(), *oc.radius_search(q, 2.0, "sphere"), *oc.knn(q, 10)]
    scarce(1 << 30)
    big = np.zeros((60_000_000, 3))  # 1.4 GB (never read)
    out_of_memory(lambda: capi.check(L.oct_set_points(oc.handle, big.ctypes.data, len(big), 0), oc.handle))
    got = [*oc.sorted_points(), *oc.radius_search(q, 2.0, "sphere"), *oc.knn(q, 10)]
    assert all(np.array_equal(a, b) for a, b in zip(want, got))
    # points that were given but not sorted are gone with the failure: an empty cloud, not a stale one
    capi.check(L.oct_set_points(oc.handle, xyz.ctypes.data, len(xyz), 0), oc.handle)
    out_of_memory(lambda: capi.check(L.oct_set_points(oc.handle, big.ctypes.data, len(big), 0), oc.handle))
    info = capi.OctTreeInfo()
    capi.check(L.oct_encode_sort(oc.handle, None, None, None, None, 0), oc.handle)
    capi.check(L.oct_build(oc.handle, C.byref(info)), oc.handle)
    assert info.n_points == 0
    oc.close()


def test_sorted_points_and_trees_that_do_not_fit(scarce):
    """Their arrays replace the cloud's one by one: a failure among them leaves no cloud, and says so."""
    from octrees_benchmark_b200 import LinearOctree, capi

    L = capi.lib()
    n = 16_000_000
    rng = np.random.default_rng(1)
    big = LinearOctree(rng.random((n, 3)), max_points_leaf=4096)
    ck = big.checkpoint()
    big.close()
    xyz = lidar_tile(50_000, 70.0, seed=4)
    q = xyz[::50].copy()
    clouds = [LinearOctree(xyz, encoder=int(ck["encoder"]), max_points_leaf=4096) for _ in range(2)]
    want = clouds[0].knn(q, 10)
    kinds = dict(box="f8", keys="u8", perm="u4", sorted_xyz="f8", offsets="u4", ranges="u8", centers="f8", radii="f8",
                 half="f8")
    arrays = {k: np.ascontiguousarray(ck[k], t) for k, t in kinds.items()}
    ptr = {k: a.ctypes.data for k, a in arrays.items()}
    info = capi.OctTreeInfo(*(int(v) for v in ck["info"]))
    scarce(512 << 20)  # 32 bytes a point with the first, 36 with the second
    calls = (lambda h: L.oct_set_sorted_points(h, ptr["sorted_xyz"], ptr["keys"], n, ptr["box"], 0),
             lambda h: L.oct_tree_import(h, C.byref(info), *ptr.values(), 0))
    for oc, call in zip(clouds, calls):
        out_of_memory(lambda: capi.check(call(oc.handle), oc.handle))
        with pytest.raises(capi.OctError) as e:
            oc.knn(q, 10)
        assert e.value.status == capi.OCT_ERR_STATE
        capi.check(L.oct_set_points(oc.handle, xyz.ctypes.data, len(xyz), 0), oc.handle)
        capi.check(L.oct_encode_sort(oc.handle, None, None, None, None, 0), oc.handle)
        capi.check(L.oct_build(oc.handle, None), oc.handle)
        assert all(np.array_equal(a, b) for a, b in zip(want, oc.knn(q, 10)))
        oc.close()


def test_ranges_without_room_for_result_chunks(scarce):
    from octrees_benchmark_b200 import LinearOctree, capi

    import torch

    L = capi.lib()
    xyz = lidar_tile(100_000, 100.0, seed=4)
    q = np.tile(xyz[:1_000], (2_000, 1))  # 2M centres: 1.6 GB of chunks
    oc = LinearOctree(xyz, max_points_leaf=64)
    oc.set_search_config(two_pass=True)
    want = oc.neighborsStruct(q, 0.4), oc.neighborsApprox(q, 0.4, 4, True)
    oc.set_search_config()
    scarce(1 << 30)
    for w, g in zip(want, (oc.neighborsStruct(q, 0.4), oc.neighborsApprox(q, 0.4, 4, True))):
        assert all(np.array_equal(a, b) for a, b in zip(w, g))
    # a call that asks for sizes only takes no chunks (158 MB for these centres)
    few = LinearOctree(xyz, max_points_leaf=64)
    few.radius_count(q[:200_000], 0.4)
    total, free = C.c_uint64(0), torch.cuda.mem_get_info()[0]
    st = L.oct_struct_search(few.handle, 2, q.ctypes.data, 200_000, None, 0.4, None, None, 0, C.byref(total), None, 0)
    assert st == capi.OCT_ERR_CAPACITY and total.value == want[0][0][200_000]
    assert free - torch.cuda.mem_get_info()[0] < (64 << 20)
    few.close()
    oc.close()
