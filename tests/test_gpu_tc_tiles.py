"""Tensor-core assignment at the edges of its forms: one cluster tile (an epilogue group
owns a row tile) against several, padding chunks, single and ragged row tiles, and near
ties inside one 32-cluster chunk. Responses are the FP64 evaluation's, exactly."""
import numpy as np
import pytest

from onedal_b200 import kmeans
from oracle import restated

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", [kmeans.compute_form.bf16x3, kmeans.compute_form.bf16])
@pytest.mark.parametrize("n,d,k", [(1, 3, 1), (127, 64, 31), (129, 65, 33), (40_000, 50, 20), (40_001, 20, 128),
                                   (19_000, 128, 129), (38_017, 100, 256), (19_000, 200, 256), (20_001, 64, 257)])
def test_forms_and_chunks(form, n, d, k):
    rng = np.random.default_rng(n + d + k)
    C = rng.uniform(-5, 5, (k, d)).astype(np.float32)
    X = (C[rng.integers(0, k, n)] + rng.standard_normal((n, d))).astype(np.float32)
    if k > 3:  # near ties with neighbours in the same chunk, an exact tie, and a NaN row
        X[::7] = (0.5 * (C[0] + C[1]) + 1e-4 * rng.standard_normal((len(X[::7]), d))).astype(np.float32)
        X[::11] = (C[0] + C[1] + C[2]) / 3
        C[k - 1] = C[0]
        X[n // 2] = np.nan
    desc = kmeans.descriptor(np.float32).set_cluster_count(k).set_compute_form(form)
    got = kmeans.infer(desc, kmeans.model(C), X).get_responses().ravel()
    want, _, _ = restated.assign_f32_in_f64(X, C)
    np.testing.assert_array_equal(got, want)
