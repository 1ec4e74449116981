"""Packet radius counts: leaves that lie inside a query are counted whole, at the widths of small and large batches,
in FP64 and with the FP32 filter, against the one-query-per-group path."""
import numpy as np
import pytest

from octrees_benchmark_b200.synth import lidar_tile

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nq", [3, 20_000, 310_000])  # widths 1, 2 and 16 (counts with the FP32 filter: 32)
@pytest.mark.parametrize("leaf", [3, 32, 500])
def test_counts(nq, leaf):
    from octrees_benchmark_b200 import LinearOctree

    xyz = lidar_tile(12_000, 50.0, seed=leaf)
    rng = np.random.default_rng(nq)
    q = xyz[rng.integers(0, len(xyz), nq)] + rng.choice([0.0, 0.3, 60.0], (nq, 1), p=[0.5, 0.45, 0.05])
    r = rng.choice([0.0, 0.4, 2.0, 9.0], nq, p=[0.1, 0.5, 0.3, 0.1])
    oc = LinearOctree(xyz, max_points_leaf=leaf)
    for kernel, algo in (("sphere", "neighborsPrune"), ("circle", "neighbors"), ("cube", "neighborsPrune"),
                         ("square", "neighborsPrune"), ("cube", "neighborsStruct")):
        oc.set_search_config(packet=False)
        want = oc.radius_count(q, r, kernel, algo)
        for fp32 in (False, True):
            oc.set_search_config(packet=True, fp32_filter=fp32)
            assert np.array_equal(want, oc.radius_count(q, r, kernel, algo)), (kernel, algo, fp32)
            if nq < 100_000 and algo == "neighborsPrune":
                oc.set_search_config(packet=True, fp32_filter=fp32, two_pass=True)
                offs, _ = oc.radius_search(q, r, kernel, algo)
                assert np.array_equal(want, np.diff(offs))
    oc.close()
