"""Empty clusters take the rows with the largest squared distances, (distance descending,
row ascending): the grid-wide selection at its edges -- one candidate, as many as rows
allow, more than the shared-memory sort holds, ties at the threshold that only some rows
of may be taken, one CTA and many. Coordinates are small integers, so distances are exact
in either type and the expected rows are known without a tolerance."""
import ctypes

import numpy as np
import pytest
import torch

from onedal_b200 import _native, kmeans

pytestmark = pytest.mark.gpu


def _step(X, C, form=_native.KMB_FORM_PLAIN):
    ctx = _native.context(0)
    n, d = X.shape
    Xd, Cd = torch.from_numpy(X).cuda(), torch.from_numpy(C).cuda()
    out, lab = torch.empty_like(Cd), torch.empty(n, dtype=torch.int32, device="cuda")
    shift, ne = ctypes.c_double(), ctypes.c_int64()
    ctx.set_stream(torch.cuda.current_stream().cuda_stream)
    dtype = _native.KMB_F32 if X.dtype == np.float32 else _native.KMB_F64
    ctx.check(ctx.lib.kmb_lloyd_step(ctx.handle, dtype, Xd.data_ptr(), n, d, Cd.data_ptr(), C.shape[0],
                                     form, 0, out.data_ptr(), lab.data_ptr(), ctypes.byref(shift),
                                     ctypes.byref(ne)))
    return out.cpu().numpy(), lab.cpu().numpy(), ne.value


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("n,m,span", [(2, 1, 9), (40, 39, 2), (5000, 1, 4), (5000, 512, 2), (5000, 1024, 40),
                                      (5000, 1025, 3), (4097, 7, 1), (700_001, 300, 3), (700_001, 3, 300)])
def test_empty_clusters_take_the_farthest_rows(dt, n, m, span):
    d = 3
    rng = np.random.default_rng(n + m)
    X = rng.integers(-span, span + 1, (n, d)).astype(dt)
    if span == 1:
        X[:] = 1  # every distance equal: the lowest rows
    C = np.zeros((m + 1, d), dt)
    C[1:] = 10000.0  # nobody's nearest
    out, lab, ne = _step(X, C)
    assert ne == m and (lab == 0).all()
    dist = (X.astype(np.int64) ** 2).sum(1)
    order = np.lexsort((np.arange(n), -dist))[:m]
    np.testing.assert_array_equal(out[1:], X[order])


def test_one_blocks_sort_outlasts_a_wait(monkeypatch):
    """65,535 empty clusters: one block sorts the candidates while the others wait, longer than
    the limit of an ordinary wait (lowered here to 2 ms); their wait allows for it."""
    n, m, d = 70_000, 65_535, 3
    rng = np.random.default_rng(9)
    X = rng.integers(-200, 201, (n, d)).astype(np.float32)
    C = np.zeros((m + 1, d), np.float32)
    C[1:] = 10000.0
    monkeypatch.setenv("KMB_GRID_WAIT_LIMIT_CYCLES", "4000000")
    out, lab, ne = _step(X, C)
    assert ne == m and (lab == 0).all()
    order = np.lexsort((np.arange(n), -(X.astype(np.int64) ** 2).sum(1)))[:m]
    np.testing.assert_array_equal(out[1:], X[order])


@pytest.mark.parametrize("n,m", [(40, 39), (300, 5), (5000, 60), (70_000, 300)])
@pytest.mark.parametrize("dt,form", [(np.float32, _native.KMB_FORM_PLAIN), (np.float64, _native.KMB_FORM_PLAIN),
                                     (np.float32, _native.KMB_FORM_BF16X3)])
def test_rows_with_a_nan_come_last(dt, form, n, m):
    """A NaN row's distance is no number: it reseeds a cluster only when no other row is left, in
    an update of the separate kernels and in a small train."""
    d = 5
    rng = np.random.default_rng(n)
    X = rng.integers(-100, 101, (n, d)).astype(dt)
    nan_rows = np.array([0, 7, n // 2, n - 1])
    X[nan_rows, [0, 1, 2, 3]] = np.array([1, -1, 1, -1]) * np.nan
    C = np.full((m + 1, d), 10000, dt)
    C[0] = 0
    dist = (X.astype(np.float64) ** 2).sum(1)
    order = np.lexsort((np.arange(n), -np.where(np.isnan(dist), -1, dist)))[:m]
    out, lab, ne = _step(X, C, form)
    assert ne == m and (lab == 0).all()
    np.testing.assert_array_equal(out[1:], X[order])
    if form == _native.KMB_FORM_PLAIN and m < 256:
        desc = kmeans.descriptor(dt).set_cluster_count(m + 1).set_max_iteration_count(1).set_compute_form(form)
        np.testing.assert_array_equal(kmeans.train(desc, X, C).get_model().get_centroids()[1:], X[order])
