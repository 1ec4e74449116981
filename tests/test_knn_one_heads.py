"""k = 1 takes every 64th query as a head: the other queries are enumerated in order (CPU restatement of
k_knn_group's index math), and single and batched searches of k = 1 around that stride give the list kernel's."""
import os
import re

import numpy as np
import pytest

S = 64


def test_stride_in_the_source():
    src = open(os.path.join(os.path.dirname(__file__), "..", "octrees_benchmark_b200", "csrc", "knn_search.cu")).read()
    assert 1 << int(re.search(r"kHeadBitsOne = (\d+);", src).group(1)) == S


@pytest.mark.parametrize("packets", [0, 1, 2, 63, 64, 65, 127, 128, 129, 4096, 4097])
def test_slots_enumerate_the_non_heads(packets):
    n_heads = (packets + S - 1) >> 6
    groups = [s + s // (S - 1) + 1 for s in range(packets - n_heads)]
    assert groups == [g for g in range(packets) if g % S]


@pytest.mark.gpu
def test_one_neighbour():
    import torch

    from octrees_benchmark_b200 import LinearOctree
    from octrees_benchmark_b200.engine import BatchEngine, Request
    from octrees_benchmark_b200.synth import lidar_tile

    xyz = lidar_tile(60_000, 100.0, seed=5)
    rng = np.random.default_rng(6)
    oc = LinearOctree(xyz, max_points_leaf=32)
    sizes = (1, 15, 17, 63, 64, 65, 129, 5_000, 200_000)
    qs = [xyz[rng.integers(0, len(xyz), n)] + rng.choice([0.0, 0.4], (n, 1)) for n in sizes]
    oc.set_search_config(packet=False)
    want = [oc.knn(q, 1) for q in qs]
    oc.set_search_config(packet=True)
    for q, w in zip(qs, want):
        assert all(np.array_equal(a, b) for a, b in zip(w, oc.knn(q, 1)))
    e = BatchEngine()
    reqs = [Request(oc, "knn", torch.from_numpy(q).cuda(), k=1) for q in qs]
    mixed = reqs + [Request(oc, "knn", torch.from_numpy(qs[4]).cuda(), k=7)]  # one group of k = 1 and 7
    for batch in (reqs, mixed, reqs):
        for p, r, w in zip(e.run(batch), batch, want):
            assert all(np.array_equal(a, b) for a, b in zip(w, e.knn_result(p, 1)))
    e.close()
    oc.close()
