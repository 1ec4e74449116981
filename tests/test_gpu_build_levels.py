"""The octree built from the keys' shared levels against the oracle, at point counts around its rows (32 keys),
warps (256) and blocks (2048) and leaf sizes from 1 to more than the cloud, with equal keys across their edges."""
import numpy as np
import pytest

from octrees_benchmark_b200.synth import lidar_tile
from tests.parity import same_f64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 255, 256, 257, 2047, 2048, 2049, 4097, 30_000])
@pytest.mark.parametrize("leaf", [1, 3, 31, 64, 5_000])
def test_levels_match_oracle(port, n, leaf):
    from octrees_benchmark_b200 import LinearOctree

    xyz = lidar_tile(n, max(1.0, 0.4 * np.sqrt(n)), seed=n + leaf)
    if n > 200:
        xyz[n // 3: n // 3 + 90] = xyz[n // 3]  # equal keys, more than a leaf of the small sizes holds
    for enc in (1, 5):
        keys, _, box, _ = port.encode_sort(enc, xyz)
        t = port.build(enc, keys, leaf, box)
        oc = LinearOctree(xyz, encoder=enc, max_points_leaf=leaf)
        assert (oc.n_total, oc.n_leaf, oc.n_internal, oc.max_depth_seen) == (t.n_total, t.n_leaf, t.n_total - t.n_leaf,
                                                                             t.max_depth)
        got, want = oc.export(), t.arrays()
        assert np.array_equal(got["offsets"], want["offsets"]) and np.array_equal(got["ranges"], want["ranges"])
        assert same_f64(got["centers"], want["centers"])
        oc.close()
