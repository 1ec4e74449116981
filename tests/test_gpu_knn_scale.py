"""kNN (collecting search) on clouds far from FP32's range, where squared distances are FP32 denormals, zeros or
FP64 denormals, and on neighbours much closer than the rounding of a wide box's octants: the list kernel's results."""
import numpy as np
import pytest

from octrees_benchmark_b200.synth import lidar_tile

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tile():
    return lidar_tile(30_000, 80.0, seed=7)


def compare(xyz, q, leaf, ks=(1, 10, 70)):
    from octrees_benchmark_b200 import LinearOctree

    for enc in (1, 5):
        oc = LinearOctree(xyz, encoder=enc, max_points_leaf=leaf)
        for k in ks:
            oc.set_search_config(packet=False)
            want = oc.knn(q, k)
            for cfg in (dict(), dict(knn_bucket=0), dict(knn_group_run=64)):
                oc.set_search_config(packet=True, **cfg)
                got = oc.knn(q, k)
                assert all(np.array_equal(a, b) for a, b in zip(want, got)), (enc, k, cfg)
        oc.close()


@pytest.mark.parametrize("scale", [1e-18, 1e-20, 1e-22, 1e-24, 1e-100, 1e-155, 1e-161, 1e24, 1e150])
@pytest.mark.parametrize("nq", [600, 40_000])
def test_scaled_tile(tile, scale, nq):
    rng = np.random.default_rng(nq)
    q = tile[rng.integers(0, len(tile), nq)] + rng.choice([0.0, 0.3], (nq, 1))
    compare(tile * scale, q * scale, 16)


@pytest.mark.parametrize("scale", [1e-20, 1e-22, 1e-24, 1e-30])
def test_runs_across_octant_faces(scale):
    """Dense centres around octant faces: a run's next ball leaves the octant that held the one before it."""
    xyz = lidar_tile(300_000, 260.0, seed=7)
    rng = np.random.default_rng(1)
    nq = 400_000
    lo, hi = xyz.min(0), xyz.max(0)
    q = xyz[rng.integers(0, len(xyz), nq)]
    cell = (hi - lo) / 32
    for a in (0, 1):
        at = rng.random(nq) < 0.5
        face = lo[a] + np.round((q[:, a] - lo[a]) / cell[a]) * cell[a]
        q[at, a] = face[at] + rng.normal(0.0, 0.4, nq)[at]
    compare(xyz * scale, q * scale, 16, ks=(1, 2))


@pytest.mark.parametrize("step", [1e-9, 1e-11, 1e-13, 1e-15])
def test_neighbours_below_the_rounding_of_the_box(step):
    """Points a few steps apart around the middle of a box 2 km wide, where octant faces meet."""
    rng = np.random.default_rng(11)
    near = rng.integers(-40, 41, (6_000, 3)) * step
    xyz = np.concatenate([near, rng.uniform(-1e3, 1e3, (3_000, 3)), [[-1e3] * 3, [1e3] * 3]])
    q = np.concatenate([near[:400], rng.integers(-45, 46, (400, 3)) * step + 0.25 * step])
    compare(xyz, q, 4)
