"""A batch whose radius results outgrow their arrays runs again: the kNN requests beside them, most of whose
queries go back to the sorted-list kernels (more equal distances than a search holds), still match single calls."""
import numpy as np
import pytest

from octrees_benchmark_b200.synth import lidar_tile

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph", [True, False])
@pytest.mark.parametrize("one_cloud", [True, False])
def test_rerun_repeats_the_handed_back_queries(graph, one_cloud):
    import torch

    from octrees_benchmark_b200 import LinearOctree
    from octrees_benchmark_b200.engine import BatchEngine, Request

    rng = np.random.default_rng(8)
    xyz = lidar_tile(400, 30.0, seed=1)
    xyz = np.concatenate([np.repeat(xyz[:20], 2_500, axis=0), xyz])
    ties = LinearOctree(xyz, max_points_leaf=64)
    tile = ties if one_cloud else LinearOctree(lidar_tile(40_000, 60.0, seed=2), max_points_leaf=64)
    reqs, want = [], []
    # more than the 64 results a centre that the first result array has room for
    r = 1.0 if one_cloud else 9.0
    centres = np.ascontiguousarray(ties.sorted_points()[2][::25][:2_000] if one_cloud else
                                   tile.sorted_points()[2][::20])
    reqs.append(Request(tile, "radius", torch.from_numpy(centres).cuda(), radius=r))
    want.append(tile.radius_search(centres, r, "sphere", "neighborsPrune"))
    assert want[0][1].shape[0] > (1 << 20)
    for k in (20, 50, 100, 250, 500, 1_000):  # every kNN variant of a batch
        q = np.ascontiguousarray(xyz[rng.integers(0, 50_000, 300)])
        reqs.append(Request(ties, "knn", torch.from_numpy(q).cuda(), k=k))
        want.append(ties.knn(q, k))
    e = BatchEngine(graph=graph)
    for _ in range(2):  # grown by the first batch, room enough for the second
        places = e.run(reqs)
        offs, idx = e.radius_result(places[0])
        assert np.array_equal(offs, want[0][0]) and np.array_equal(idx, want[0][1])
        for r, p, w in zip(reqs[1:], places[1:], want[1:]):
            got = e.knn_result(p, r.k)
            assert all(np.array_equal(a, b) for a, b in zip(got, w)), r.k
    e.close()
