"""Failure paths, exercised without faulting the GPU.

* A bounded device wait that runs out: the tensor-core kernel's pipeline waits
  get a short limit (KMB_TC_WAIT_LIMIT_CYCLES, read at launch); the launch must
  drain its own copies and MMAs, report KMB_ETIMEDOUT, and leave the context
  usable for a correct call afterwards.
* A grid barrier's wait that runs out (KMB_GRID_WAIT_LIMIT_CYCLES, read at launch): the
  small train, the update's last launch and the sharded train's candidate selection
  report KMB_ETIMEDOUT, and the context trains correctly afterwards.
* Host-side allocation failure (KMB_FAIL_ALLOC=1 makes every workspace growth
  fail): KMB_ENOMEM, raised as bad_alloc by the Python mirror and as oneDAL's
  host_bad_alloc by the dispatcher (backend/interop/error_converter.cpp maps
  DAAL's allocation errors the same way); the next call without the hook works.
* NaN rows: the reference's argmin starts from the first cluster's score and
  replaces it only on a strictly smaller one (kmeans_lloyd_impl.i:197-216,
  kmeans_lloyd_postprocessing.h:95-130), so a row whose scores are all NaN gets
  cluster 0; the other rows are unaffected.
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest
import torch

from onedal_b200 import _native, kmeans
from oracle import restated

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CLIENT = os.path.join(ROOT, "integration", "_build", "kmeans_client")


def _blobs(n, d, k, seed):
    rng = np.random.default_rng(seed)
    centres = rng.uniform(-5, 5, (k, d))
    X = (centres[rng.integers(0, k, n)] + rng.standard_normal((n, d))).astype(np.float32)
    return X, X[rng.choice(n, k, replace=False)].copy()


@pytest.mark.parametrize("form", [kmeans.compute_form.bf16x3, kmeans.compute_form.bf16])
def test_tensor_core_wait_limit_reports_timeout_and_context_recovers(form, monkeypatch):
    X, C = _blobs(60000, 128, 512, 31)
    desc = kmeans.descriptor(np.float32).set_cluster_count(512).set_compute_form(form)
    monkeypatch.setenv("KMB_TC_WAIT_LIMIT_CYCLES", "200")  # below one accumulator's MMA time
    with pytest.raises(kmeans.internal_error) as err:
        kmeans.infer(desc, kmeans.model(C), X)
    assert "status 4" in str(err.value)  # KMB_ETIMEDOUT
    monkeypatch.delenv("KMB_TC_WAIT_LIMIT_CYCLES")
    r = kmeans.infer(desc, kmeans.model(C), X)
    lab64, _, _ = restated.assign_f32_in_f64(X, C)
    np.testing.assert_array_equal(r.get_responses().ravel(), lab64)
    t = kmeans.train(desc.set_max_iteration_count(3), X, C)
    assert t.get_iteration_count() == 3


def _train(dt, n, k, T):
    rng = np.random.default_rng(n)
    X = torch.from_numpy(rng.standard_normal((n, 20)).astype(dt)).cuda()
    C = X[:k].clone()
    C[-3:] = 1e4  # nobody's nearest
    desc = kmeans.descriptor(dt).set_cluster_count(k).set_max_iteration_count(T)
    desc.set_compute_form(kmeans.compute_form.plain)

    def run():
        r = kmeans.train(desc, X, C)
        return r.get_model().get_centroids(), r.get_responses()
    return run


def _train_sharded(dt, n, k, T):
    rng = np.random.default_rng(n)
    X = torch.from_numpy(rng.standard_normal((n, 20)).astype(dt)).cuda()
    C0 = X[:k].clone()
    C0[-3:] = 1e4
    gather = _native.ALLGATHER_FN(lambda _u, send, nbytes, recv: ctypes.memmove(recv, send, nbytes) and 0)
    comm = _native.kmb_communicator(None, 0, 1, _native.ALLREDUCE_F64_FN(lambda _u, _b, _c: 0), gather)
    p = _native.kmb_params(k, T, 0.0, _native.KMB_FORM_PLAIN, 0)

    def run():
        ctx = _native.context(0)
        ctx.set_stream(torch.cuda.current_stream().cuda_stream)
        C, lab = torch.empty_like(C0), torch.empty(n, dtype=torch.int32, device="cuda")
        obj, it = ctypes.c_double(), ctypes.c_int64()
        ctx.check(ctx.lib.kmb_train_spmd(ctx.handle, _native.KMB_F32 if dt == np.float32 else _native.KMB_F64,
                                         X.data_ptr(), n, 20, C0.data_ptr(), ctypes.byref(p), ctypes.byref(comm),
                                         C.data_ptr(), lab.data_ptr(), ctypes.byref(obj), ctypes.byref(it)))
        return C, lab
    return run


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("make,n,k", [(_train, 8_000, 40), (_train, 600_000, 300), (_train_sharded, 600_000, 40)],
                         ids=["small", "update_tail", "sharded"])
def test_grid_wait_limit_reports_timeout_and_context_recovers(make, n, k, dt, monkeypatch):
    run = make(dt, n, k, 2)
    monkeypatch.setenv("KMB_GRID_WAIT_LIMIT_CYCLES", "1")  # the CTAs do not all arrive within a poll
    with pytest.raises((kmeans.internal_error, _native.NativeError)) as err:
        run()
    assert "status 4" in str(err.value)  # KMB_ETIMEDOUT
    monkeypatch.delenv("KMB_GRID_WAIT_LIMIT_CYCLES")
    got = run()
    _native.context(0).lib.kmb_context_release_workspace(_native.context(0).handle)  # state as in a new context
    for a, b in zip(got, run()):
        assert torch.equal(a, b)


def test_allocation_failure_raises_bad_alloc_and_context_recovers(monkeypatch):
    X, C = _blobs(30000, 24, 40, 32)
    desc = kmeans.descriptor(np.float32).set_cluster_count(40).set_max_iteration_count(5)
    _native.context(0).lib.kmb_context_release_workspace(_native.context(0).handle)
    monkeypatch.setenv("KMB_FAIL_ALLOC", "1")
    with pytest.raises(kmeans.bad_alloc):
        kmeans.train(desc, X, C)
    monkeypatch.delenv("KMB_FAIL_ALLOC")
    r = kmeans.train(desc, X, C)
    ref = restated.train(X.astype(np.float64), C.astype(np.float64), 5, 0.0)
    assert r.get_iteration_count() == ref[3]


@pytest.mark.skipif(not os.path.exists(CLIENT), reason="integration client not built")
def test_client_maps_allocation_failure_to_host_bad_alloc(tmp_path):
    """Through dal::train: KMB_ENOMEM becomes oneDAL's host_bad_alloc, whose what()
    is std::bad_alloc's (cpp/oneapi/dal/exceptions.cpp:61-63)."""
    import json
    g = json.load(open(os.path.join(ROOT, "tests", "golden", "gold.json")))
    X = np.asarray(g["data"], np.float64).ravel()
    C = np.asarray(g["initial_centroids"], np.float64).ravel()
    p = tmp_path / "gold.txt"
    p.write_text("%d %d %d\n%s\n%s\n" % (g["row_count"], g["column_count"], g["cluster_count"],
                                          " ".join(repr(float(v)) for v in X), " ".join(repr(float(v)) for v in C)))
    env = dict(os.environ, KMB_FAIL_ALLOC="1")
    r = subprocess.run([CLIENT, str(p), "double"], capture_output=True, text=True, timeout=120, env=env)
    assert r.returncode == 1, (r.stdout, r.stderr)
    assert r.stdout.strip() == "exception: std::bad_alloc", r.stdout


@pytest.mark.parametrize("dt,form", [(np.float32, kmeans.compute_form.plain), (np.float64, kmeans.compute_form.plain),
                                     (np.float32, kmeans.compute_form.bf16x3)])
def test_nan_rows_take_cluster_zero(dt, form):
    X, C = _blobs(5000, 32, 17, 33)
    X = X.astype(dt)
    C = C.astype(dt)
    nan_rows = np.array([3, 100, 4999])
    X[nan_rows, 5] = np.nan
    desc = kmeans.descriptor(dt).set_cluster_count(17).set_compute_form(form)
    r = kmeans.infer(desc, kmeans.model(C), X)
    lab = r.get_responses().ravel()
    oracle_lab, _ = restated.infer(X.astype(np.float64), C.astype(np.float64), False)
    assert (oracle_lab[nan_rows] == 0).all()
    np.testing.assert_array_equal(lab, oracle_lab)
