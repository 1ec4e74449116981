"""kNN (collecting search) of centres far from the cloud, where all distances and node bounds are nearly one: the
results of the per-query search, in about the time that centres at the cloud take."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def knn_ms(oc, q, k):
    """Median device time of a search with device buffers."""
    import torch

    from octrees_benchmark_b200 import capi

    q = torch.from_numpy(np.ascontiguousarray(q)).cuda()
    idx = torch.zeros((len(q), k), dtype=torch.int32, device="cuda")
    d2 = torch.zeros((len(q), k), dtype=torch.float64, device="cuda")
    ts = []
    for _ in range(8):
        torch.cuda.synchronize()
        start, end = torch.cuda.Event(True), torch.cuda.Event(True)
        start.record()
        capi.check(capi.lib().oct_knn(oc.handle, q.data_ptr(), len(q), k, idx.data_ptr(), d2.data_ptr(), None,
                                      capi.OCT_MEM_DEVICE), oc.handle, "oct_knn")
        end.record()
        end.synchronize()
        ts.append(start.elapsed_time(end))
    return float(np.median(ts[1:]))


@pytest.fixture(scope="module")
def cube():
    return np.random.default_rng(3).uniform(0.0, 100.0, (500_000, 3))


@pytest.mark.parametrize("k", [64, 250, 1000])
@pytest.mark.parametrize("away", [1.5, 1e3, 1e9])
def test_far_centres(cube, k, away):
    from octrees_benchmark_b200 import LinearOctree

    rng = np.random.default_rng(k)
    xyz = cube[:60_000]
    q = xyz[rng.integers(0, len(xyz), 200)] + 100.0 * away * rng.uniform(-1.0, 1.0, (200, 3))
    oc = LinearOctree(xyz, encoder=5, max_points_leaf=16)
    got = oc.knn(q, k)
    oc.set_search_config(packet=False)
    want = oc.knn(q, k)
    assert all(np.array_equal(a, b) for a, b in zip(want, got))


def test_time_of_long_lists_far_away(cube):
    """k = 1000 beside a cube: 3.7 and 6.7 times the time of centres in it while the far half of the open nodes was
    chosen by halves of the largest bound, which dropped all of them; 1.2 times since."""
    import torch

    from octrees_benchmark_b200 import LinearOctree

    rng = np.random.default_rng(4)
    at = cube[rng.integers(0, len(cube), 300)]
    oc = LinearOctree(cube, encoder=5, max_points_leaf=64, stream=torch.cuda.current_stream().cuda_stream)
    inside = knn_ms(oc, at, 1000)
    beside = knn_ms(oc, at + [150.0, 0.0, 0.0], 1000)
    around = knn_ms(oc, at + 200.0 * rng.uniform(-1.0, 1.0, at.shape), 1000)
    assert max(beside, around) < 2.5 * inside, (inside, beside, around)


@pytest.mark.parametrize("k", [1, 10, 70])
@pytest.mark.parametrize("share", [0.02, 0.5, 1.0])
def test_centres_outside_the_box(cube, k, share):
    """Batches that seed, with centres outside the box among them, alone and in a batch of two clouds."""
    import torch

    from octrees_benchmark_b200 import LinearOctree
    from octrees_benchmark_b200.engine import BatchEngine, Request

    rng = np.random.default_rng(k)
    clouds = [cube[:40_000], cube[:30_000] * [1.0, 1.0, 0.0]]
    ocs = [LinearOctree(xyz, encoder=enc, max_points_leaf=16) for xyz, enc in zip(clouds, (1, 5))]
    reqs, want = [], []
    for xyz, oc in zip(clouds, ocs):
        q = xyz[rng.integers(0, len(xyz), 30_000)]
        out = rng.random(len(q)) < share
        q[out] += rng.uniform(-150.0, 150.0, (int(out.sum()), 3))
        got = oc.knn(q, k)
        oc.set_search_config(packet=False)
        want.append(oc.knn(q, k))
        oc.set_search_config(packet=True)
        assert all(np.array_equal(a, b) for a, b in zip(want[-1], got))
        reqs.append(Request(oc, "knn", torch.from_numpy(q).cuda(), k=k))
    engine = BatchEngine()
    places = engine.run(reqs)
    for p, w in zip(places, want):
        got = engine.knn_result(p, k)
        assert all(np.array_equal(a, b) for a, b in zip(w, got))


@pytest.mark.parametrize("flat", [False, True])
def test_time_of_large_batches_outside_the_box(cube, flat):
    """A batch that seeds takes about the time of one whose centres all start cold (knn_estimate -1); outside the box
    2.7 and 3.7 times that while those centres were seeded too."""
    import torch

    from octrees_benchmark_b200 import LinearOctree

    rng = np.random.default_rng(5)
    xyz = cube * [1.0, 1.0, 0.0] if flat else cube
    q = xyz[rng.integers(0, len(xyz), 20_000)] + ([150.0, 0.0, 0.0] if flat else rng.uniform(-200.0, 200.0, (20_000, 3)))
    oc = LinearOctree(xyz, encoder=5, max_points_leaf=64, stream=torch.cuda.current_stream().cuda_stream)
    seeded = knn_ms(oc, q, 10)
    oc.set_search_config(knn_estimate=-1)
    cold = knn_ms(oc, q, 10)
    assert seeded < 1.6 * cold, (seeded, cold)
