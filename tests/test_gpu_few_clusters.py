"""Few clusters, rows through a warp's tile and read directly: integer rows, whose scores are
exact in both types, so every label is the FP64 evaluation's; by infer, and by a train of no
iterations with the recheck, whose queue the kernel then fills. Part tiles, one row, rows past
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
    Xd, Cd = buf[1:].view(n, d), torch.from_numpy(C).cuda()
    got = kmeans.infer(desc, kmeans.model(Cd), Xd).get_responses()
    np.testing.assert_array_equal(got.cpu().numpy().ravel(), np.asarray(want).ravel())
    if n < k:
        return  # (a train has at least as many rows as clusters)
    t = kmeans.train(desc.set_recheck(True).set_max_iteration_count(0), Xd, Cd)
    np.testing.assert_array_equal(t.get_responses().cpu().numpy().ravel(), np.asarray(want).ravel())
    # the queue holds every row whose two nearest clusters tie, and no row that is clear of
    # the band: scores are whole or half numbers, the band is far below a half
    s = 0.5 * (C.astype(np.float64) ** 2).sum(1) - X.astype(np.float64) @ C.astype(np.float64).T
    two = np.partition(s, 1, axis=1)[:, :2] if k > 1 else np.column_stack([s[:, 0], s[:, 0] + 1])
    assert t.stats.rechecked_rows == (two[:, 0] == two[:, 1]).sum()
