"""Few clusters, rows through a warp's tile and read directly: integer rows, whose scores are
exact in both types, so every label is the FP64 evaluation's. Part tiles, one row, rows past
one pass of the grid, the narrowest and widest rows of each form, part groups of clusters, a
base that is only element aligned."""
import numpy as np
import pytest
import torch

from onedal_b200 import kmeans
from oracle import restated

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("n,d,k", [(1, 33, 1), (31, 64, 2), (33, 63, 3), (129, 47, 4), (1000, 64, 5), (5001, 33, 32),
                                   (148 * 16 * 128 + 77, 34, 9), (4000, 32, 31), (4000, 1, 6)])
def test_labels(dt, n, d, k):
    rng = np.random.default_rng(n + d + k)
    X = rng.integers(-12, 13, (n, d)).astype(dt)
    C = rng.integers(-12, 13, (k, d)).astype(dt)
    buf = torch.zeros(X.size + 1, dtype=torch.from_numpy(X).dtype, device="cuda")
    buf[1:] = torch.from_numpy(X).cuda().reshape(-1)
    desc = kmeans.descriptor(dt).set_cluster_count(k).set_compute_form(kmeans.compute_form.plain)
    want, _ = restated.infer(X.astype(np.float64), C.astype(np.float64), True)
    for recheck in (False, True):
        got = kmeans.infer(desc.set_recheck(recheck), kmeans.model(torch.from_numpy(C).cuda()), buf[1:].view(n, d))
        np.testing.assert_array_equal(got.get_responses().cpu().numpy().ravel(), np.asarray(want).ravel())
