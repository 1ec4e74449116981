"""Clouds created, searched and destroyed on several threads, on idle streams and a caller's, with memory trimmed
between: every iteration of every thread is counted, and what it raises is kept."""
import threading
import traceback

import numpy as np
import pytest

from octrees_benchmark_b200.synth import lidar_tile

pytestmark = pytest.mark.gpu


def test_every_iteration_of_every_thread():
    import torch

    from octrees_benchmark_b200 import LinearOctree, capi

    xyz = [lidar_tile(n, 45.0, seed=2) for n in (300, 8_000, 30_000)]
    want = [LinearOctree(x).knn(x[:50], 5) for x in xyz]
    done, errors = [], []

    def work(t):
        try:
            s = torch.cuda.Stream()
            for i in range(25):
                x, w = xyz[(i + t) % 3], want[(i + t) % 3]
                oc = LinearOctree(x, stream=s.cuda_stream if (i + t) % 4 == 0 else None)
                got = oc.knn(x[:50], 5)
                assert all(np.array_equal(a, b) for a, b in zip(w, got)), (t, i)
                if i % 5 == 4:  # other points on the same handle
                    capi.check(oc._L.oct_set_points(oc.handle, x.ctypes.data, len(x) // 2, 0), oc.handle)
                    capi.check(oc._L.oct_encode_sort(oc.handle, None, None, None, None, 0), oc.handle)
                oc.close()
                if i % 10 == 9:
                    capi.check(capi.lib().oct_trim_cloud_memory(0))
                done.append((t, i))
        except BaseException:
            errors.append(traceback.format_exc())

    threads = [threading.Thread(target=work, args=(t,)) for t in range(6)]
    [t.start() for t in threads]
    [t.join(120) for t in threads]
    assert not errors, errors[0]
    assert len(done) == 6 * 25
