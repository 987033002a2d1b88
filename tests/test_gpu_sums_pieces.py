"""The counting sort and the per-piece sums around the row counts where a chunk's and a
piece's rows change: integer rows, whose sums are exact in any order, so a centroid is one
rounded division away from the exact sum over its rows."""
import numpy as np
import pytest
import torch

from onedal_b200 import kmeans

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("n", [127, 129, 257, 606_207, 606_208, 1_212_415, 1_212_417, 2_424_831, 2_424_833])
@pytest.mark.parametrize("k", [2, 257])
def test_sums(dt, n, k):
    if k > n:
        pytest.skip("more clusters than rows")
    rng = np.random.default_rng(n + k)
    # every row near 0 for a while, then spread: long runs of one cluster and ragged last pieces
    X = rng.integers(-500, 501, (n, 3))
    X[: n // 3] //= 100
    C0 = X[rng.permutation(n)[:k]].astype(dt) + dt(0.25)
    Xd, Cd = torch.from_numpy(X.astype(dt)).cuda(), torch.from_numpy(C0).cuda()
    desc = kmeans.descriptor(dt).set_cluster_count(k).set_max_iteration_count(1)
    desc.set_compute_form(kmeans.compute_form.plain).set_recheck(True)
    got = kmeans.train(desc, Xd, Cd)
    lab = kmeans.infer(desc, kmeans.model(Cd), Xd).get_responses().cpu().numpy().ravel()
    count = np.bincount(lab, minlength=k)
    sums = np.stack([np.bincount(lab, weights=X[:, t], minlength=k) for t in range(3)], 1)
    full = count > 0
    want = (sums[full] / count[full, None]).astype(dt)
    # one division (correctly rounded or not) and one rounding to the type: one unit each
    np.testing.assert_allclose(got.get_model().get_centroids().cpu().numpy()[full], want, rtol=2 * np.finfo(dt).eps, atol=0)
