"""Packet radius searches at the batch sizes where the packet width changes, against the plain path."""
import numpy as np
import pytest

from octrees_benchmark_b200.synth import lidar_tile

pytestmark = pytest.mark.gpu

SIZES = (1, 3, 4095, 4097, 18_943, 18_945, 37_889, 75_777, 151_553)  # widths 1, 2, 4, 8, 16 on 148 SMs


@pytest.fixture(scope="module")
def cloud():
    from octrees_benchmark_b200 import LinearOctree

    xyz = lidar_tile(60_000, 120.0, seed=9)
    return xyz, LinearOctree(xyz, encoder=5, max_points_leaf=32)


@pytest.mark.parametrize("nq", SIZES)
@pytest.mark.parametrize("kernel,algo", [("sphere", "neighborsPrune"), ("square", "neighbors")])
def test_packet_width(cloud, nq, kernel, algo):
    xyz, oc = cloud
    q = xyz[np.random.default_rng(nq).integers(0, len(xyz), nq)] + 0.25
    r = np.random.default_rng(nq + 1).uniform(0.1, 1.5, nq)
    oc.set_search_config(packet=False)
    o0, i0 = oc.radius_search(q, r, kernel, algo)
    n0 = oc.neighborsStruct(q, r, kernel)
    for two_pass in (False, True):
        oc.set_search_config(packet=True, two_pass=two_pass)
        o1, i1 = oc.radius_search(q, r, kernel, algo)
        assert np.array_equal(o0, o1) and np.array_equal(i0, i1)
    for a, b in zip(n0, oc.neighborsStruct(q, r, kernel)):
        assert np.array_equal(a, b)
