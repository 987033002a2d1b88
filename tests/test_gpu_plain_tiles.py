"""Plain assignment at the tile edges of its FP64 and few-row kernels: integer coordinates,
so every score is exact in either type, the nearest cluster is known, ties go to the lowest
index, and the FP64 recheck changes nothing."""
import numpy as np
import pytest

from onedal_b200 import kmeans

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("n,d,k", [(1, 1, 33), (31, 7, 64), (33, 8, 65), (129, 17, 128), (128, 65, 129), (1000, 33, 191),
                                   (257, 96, 300), (4097, 64, 257), (20_100, 12, 513), (130, 300, 40)])
def test_exact_scores(dt, n, d, k):
    rng = np.random.default_rng(n + d + k)
    C = rng.integers(-8, 9, (k, d))
    C[k // 2] = C[0]  # an exact tie between two tiles
    X = C[rng.integers(0, k, n)] + rng.integers(-2, 3, (n, d))
    score = (C * C).sum(1) - 2 * X @ C.T  # twice the scores, in integers
    want = score.argmin(1)
    desc = kmeans.descriptor(dt).set_cluster_count(k).set_compute_form(kmeans.compute_form.plain)
    r = kmeans.infer(desc, kmeans.model(C.astype(dt)), X.astype(dt))
    np.testing.assert_array_equal(r.get_responses().ravel(), want)
    if n >= k:
        desc.set_max_iteration_count(0).set_recheck(True)
        t = kmeans.train(desc, X.astype(dt), C.astype(dt))
        np.testing.assert_array_equal(t.get_responses().ravel(), want)
