"""The collecting kNN (packet path) against the best-first list kernel of the plain path: list lengths around
its buffer and bin sizes, clouds whose distances crowd into few bins or tie, centres far from every point."""
import numpy as np
import pytest

from octrees_benchmark_b200.synth import lidar_tile

pytestmark = pytest.mark.gpu

KS = (1, 2, 31, 32, 33, 64, 65, 128, 129, 256, 257, 513, 1024)


def clouds():
    rng = np.random.default_rng(3)
    tile = lidar_tile(9_000, 45.0, seed=4)
    grid = np.stack(np.meshgrid(np.arange(24.0), np.arange(24.0), np.arange(6.0)), -1).reshape(-1, 3)
    far = np.concatenate([rng.normal(0.0, 1e-3, (900, 3)), rng.normal(0.0, 1e-3, (700, 3)) + 4e3,
                          rng.uniform(-5e3, 5e3, (200, 3))])
    flat = rng.uniform(0.0, 60.0, (5_000, 3))
    flat[:, 2] = 7.0
    return {"tile": tile, "grid": grid, "equal": np.repeat(tile[:3], 1_200, axis=0), "far": far, "flat": flat,
            "few": tile[:40], "utm": lidar_tile(5_000, 40.0, seed=6) + np.array([4.6e6, 5.1e5, 0.0])}


@pytest.mark.parametrize("name", ["tile", "grid", "equal", "far", "flat", "few", "utm"])
@pytest.mark.parametrize("leaf", [4, 64, 3_000])
def test_collect_matches_list_kernel(name, leaf):
    from octrees_benchmark_b200 import LinearOctree

    xyz = clouds()[name]
    rng = np.random.default_rng(5)
    lo, hi = xyz.min(0), xyz.max(0)
    q = np.concatenate([xyz[rng.integers(0, len(xyz), 60)], rng.uniform(lo - 3.0, hi + 3.0, (40, 3)),
                        rng.uniform(lo, hi, (1, 3)) + 1e5])
    oc = LinearOctree(xyz, encoder=1 if leaf == 4 else 5, max_points_leaf=leaf)
    for k in KS:
        oc.set_search_config(packet=False)
        want = oc.knn(q, k)
        for cfg in (dict(), dict(knn_estimate=-1), dict(knn_bucket=0), dict(fp32_filter=True), dict(knn_group_run=64)):
            oc.set_search_config(packet=True, **cfg)
            got = oc.knn(q, k)
            assert all(np.array_equal(a, b) for a, b in zip(want, got)), (k, cfg)
    oc.close()


@pytest.mark.parametrize("nq", [17, 5_000, 40_000, 150_000])
def test_runs_and_heads(nq):
    """Batches around the sizes where runs of seeded queries begin, in curve order and at one place."""
    from octrees_benchmark_b200 import LinearOctree

    xyz = lidar_tile(30_000, 80.0, seed=7)
    rng = np.random.default_rng(nq)
    q = xyz[rng.integers(0, len(xyz), nq)] + rng.choice([0.0, 0.3, 20.0], (nq, 1), p=[0.5, 0.49, 0.01])
    oc = LinearOctree(xyz, max_points_leaf=64)
    for k in (1, 10, 70):
        oc.set_search_config(packet=False)
        want = oc.knn(q, k)
        oc.set_search_config(packet=True)
        assert all(np.array_equal(a, b) for a, b in zip(want, oc.knn(q, k))), k
    oc.close()
