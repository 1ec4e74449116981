"""Calls that run out of device memory return an error, and the calls after them answer as before."""
import numpy as np
import pytest

from octrees_benchmark_b200.synth import lidar_tile

pytestmark = pytest.mark.gpu

LEFT = 3 << 30  # bytes of device memory a test leaves free


@pytest.fixture
def scarce():
    """All of the device's memory but LEFT bytes, and the clouds' own pool, taken by the program."""
    import torch

    from octrees_benchmark_b200 import capi

    def take():
        capi.check(capi.lib().oct_trim_cloud_memory(0), None)
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        held.append(torch.empty(torch.cuda.mem_get_info()[0] - LEFT, dtype=torch.uint8, device="cuda"))

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
    scarce()
    out_of_memory(lambda: oc.radius_hash(q, 1e3, "sphere"))  # 4e9 results
    got = oc.radius_search(q, 2.0, "sphere"), oc.neighborsStruct(q, 2.0, "square"), oc.radius_hash(q, 2.0, "cube")
    for w, g in zip(want, got):
        assert all(np.array_equal(a, b) for a, b in zip(w, g))
    oc.close()
