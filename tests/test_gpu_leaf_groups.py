"""Packet searches that test several leaves as one run of points, at leaf sizes around a warp's width,
against the one-query-per-group path (ranges cut at leaf ends, runs that cross 32 points, empty octants)."""
import numpy as np
import pytest

from octrees_benchmark_b200.synth import lidar_tile

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("leaf", [1, 5, 31, 32, 33, 64, 200])
@pytest.mark.parametrize("kernel", ["sphere", "circle", "cube", "square"])
def test_leaf_groups(leaf, kernel):
    from octrees_benchmark_b200 import LinearOctree

    xyz = lidar_tile(6_000, 40.0, seed=leaf)
    xyz[100:180] = xyz[100]  # a leaf of equal points at the deepest level
    q = np.concatenate([xyz[:300] + 0.1, xyz[100:101], xyz[:1] + 1e4])
    oc = LinearOctree(xyz, encoder=1 if leaf % 2 else 5, max_points_leaf=leaf)
    for r in (0.0, 0.7, 4.0, 100.0):
        got = {}
        for packet, two_pass, fp32 in ((False, False, False), (True, False, False), (True, True, False),
                                       (True, False, True)):
            oc.set_search_config(packet=packet, two_pass=two_pass, fp32_filter=fp32)
            got[packet, two_pass, fp32] = [oc.radius_search(q, r, kernel, a) for a in ("neighbors", "neighborsPrune")] + [
                oc.neighborsStruct(q, r, kernel), oc.neighborsApprox(q, r, 3, True, kernel),
                oc.neighborsApprox(q, r, 4, False, kernel)]
        want = got.pop((False, False, False))
        for key, res in got.items():
            for w, g in zip(want, res):
                assert all(np.array_equal(x, y) for x, y in zip(w, g)), (key, r)
