"""Small dense trains in one launch against the general path, which a call takes while kernel
timing is on (float: the same arithmetic, so everything is equal bit for bit) or with the
FP64 recheck (double: at values whose near ties are exact, so that both give the same
responses). Sizes at the edges of the rule and of the
kernel: one CTA and many, ragged rows per CTA, the padded column counts, one cluster, as
many clusters as threads allow, fewer rows than clusters would fill, empty clusters over
several CTAs."""
import ctypes
import json
import time

import numpy as np
import pytest
import torch

from onedal_b200 import _native, kmeans
from oracle import restated

pytestmark = pytest.mark.gpu


def _data(n, d, k, dt, seed, dup):
    rng = np.random.default_rng(seed)
    centres = rng.integers(-40, 41, (k, d))
    X = (centres[rng.integers(0, k, n)] * 4 + rng.integers(-6, 7, (n, d))).astype(dt)
    C0 = X[rng.permutation(n)[:k]].copy()
    if dup and k > 2:
        C0[k // 2:] = C0[0]  # empty clusters in the first update
    return X, C0


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("n,d,k,T,dup", [(1, 1, 1, 3, False), (100, 3, 3, 50, False), (513, 4, 2, 20, False),
                                         (2047, 24, 7, 20, True), (2049, 33, 40, 10, True), (30_001, 20, 20, 12, False),
                                         (9_999, 64, 256, 6, True), (148 * 256 + 1, 8, 33, 9, True),
                                         (60_000, 47, 61, 5, False),
                                         # the edges of the rule: one CTA or more, rows per CTA, the general path
                                         (512, 16, 16, 8, True), (512, 16, 17, 8, False), (4096, 64, 161, 5, True),
                                         (4095, 64, 161, 5, False), (1025, 64, 160, 5, True), (3000, 32, 256, 5, False),
                                         (2500, 33, 186, 5, True), (2500, 33, 187, 5, False)])
def test_equals_the_general_path(dt, n, d, k, T, dup):
    X, C0 = _data(n, d, k, dt, n + d + k, dup)
    desc = kmeans.descriptor(dt).set_cluster_count(k).set_max_iteration_count(T)
    desc.set_compute_form(kmeans.compute_form.plain)
    a = kmeans.train(desc, X, C0)
    if dt == np.float32:
        ctx = _native.context(0)
        ctx.check(ctx.lib.kmb_context_set_kernel_timing(ctx.handle, 1))
        try:
            b = kmeans.train(desc, X, C0)
        finally:
            ctx.check(ctx.lib.kmb_context_set_kernel_timing(ctx.handle, 0))
    else:
        b = kmeans.train(desc.set_recheck(True), X, C0)
    assert a.get_iteration_count() == b.get_iteration_count()
    assert a.stats.empty_cluster_events == b.stats.empty_cluster_events
    np.testing.assert_array_equal(a.get_responses(), b.get_responses())
    if dt == np.float32:
        np.testing.assert_array_equal(a.get_model().get_centroids(), b.get_model().get_centroids())
        lab, _, _ = restated.assign_f32_in_f64(X, a.get_model().get_centroids())
        assert (a.get_responses().ravel() == lab).mean() > 0.999
    else:
        # sums in another order: n additions of values below M, 2^-53 each, over the count
        ca, cb = a.get_model().get_centroids(), b.get_model().get_centroids()
        np.testing.assert_allclose(ca, cb, rtol=0, atol=n * 2.0 ** -52 * np.abs(X).max())
    fa, fb = a.get_objective_function_value(), b.get_objective_function_value()
    assert abs(fa - fb) <= 1e-6 * max(fa, fb, 1e-300)


def test_empty_clusters_take_the_farthest_rows_over_all_blocks():
    n, d, k = 148 * 300, 3, 40
    rng = np.random.default_rng(3)
    X = rng.integers(-300, 301, (n, d)).astype(np.float64)
    X[1::2] = X[0::2]  # every distance twice: the lower row first
    C0 = np.full((k, d), 1e6)
    C0[0] = 0
    desc = kmeans.descriptor(np.float64).set_cluster_count(k).set_max_iteration_count(1)
    r = kmeans.train(desc, X, C0)
    order = np.lexsort((np.arange(n), -(X ** 2).sum(1)))[:k - 1]
    np.testing.assert_array_equal(r.get_model().get_centroids()[1:], X[order])
    assert r.stats.empty_cluster_events == k - 1


@pytest.mark.parametrize("dt,n,d,k,span", [(np.float32, 1_100_000, 3, 200, 300), (np.float32, 1_100_000, 3, 200, 2),
                                           (np.float64, 1_050_000, 1, 100, 10**6), (np.float32, 1_050_000, 1, 256, 0),
                                           (np.float64, 2000, 1, 256, 9)])
def test_empty_clusters_take_the_farthest_of_many_rows_per_block(dt, n, d, k, span):
    """Thousands of rows in a block, all but one cluster empty: distances that differ, that tie
    in their thousands, and that are all the same (the lowest rows then)."""
    rng = np.random.default_rng(span)
    X = rng.integers(-span, span + 1, (n, d)).astype(dt) + 1
    C0 = np.full((k, d), 1e9, dt)
    C0[0] = 0
    desc = kmeans.descriptor(dt).set_cluster_count(k).set_max_iteration_count(1)
    r = kmeans.train(desc.set_compute_form(kmeans.compute_form.plain), X, C0)
    order = np.lexsort((np.arange(n), -(X.astype(np.float64) ** 2).sum(1)))[:k - 1]
    np.testing.assert_array_equal(r.get_model().get_centroids()[1:], X[order])


@pytest.mark.parametrize("dt,n,d,k", [(np.float32, 1_100_000, 3, 200), (np.float64, 1_050_000, 1, 100)])
def test_an_empty_cluster_costs_no_more_than_the_iteration(dt, n, d, k):
    """The selection reads the distances a few times; ranking rows against rows took six
    trains' time."""
    g = torch.Generator(device="cuda").manual_seed(1)
    X = torch.randn(n, d, device="cuda", generator=g, dtype=torch.float32 if dt == np.float32 else torch.float64)
    desc = kmeans.descriptor(dt).set_cluster_count(k).set_max_iteration_count(1)
    desc.set_compute_form(kmeans.compute_form.plain)
    times = []
    for empty in (0, 1):
        C = X[:k].clone()
        if empty:
            C[-1] = 1e6
        assert kmeans.train(desc, X, C).stats.empty_cluster_events == empty
        runs = []
        for _ in range(9):
            t = time.perf_counter()
            kmeans.train(desc, X, C)
            runs.append(time.perf_counter() - t)
        times.append(sorted(runs)[4])
    assert times[1] < 2 * times[0], times


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("n,d,k", [(256, 64, 256), (400, 64, 256), (1000, 64, 256), (4000, 64, 256), (12_000, 1, 80)])
def test_no_slower_than_the_general_path(dt, n, d, k):
    """The general path is asked for with the recheck, which it pays for as well."""
    g = torch.Generator(device="cuda").manual_seed(1)
    X = torch.randn(n, d, device="cuda", generator=g, dtype=torch.float32 if dt == np.float32 else torch.float64)
    C = X[:k].clone()
    times = []
    for recheck in (False, True):
        desc = kmeans.descriptor(dt).set_cluster_count(k).set_max_iteration_count(10)
        desc.set_compute_form(kmeans.compute_form.plain).set_recheck(recheck)
        runs = []
        for _ in range(13):
            t = time.perf_counter()
            kmeans.train(desc, X, C)
            runs.append(time.perf_counter() - t)
        times.append(sorted(runs)[6])
    assert times[0] < 1.25 * times[1], times


@pytest.mark.parametrize("span", [1, 40, 80, 120])
def test_float_sums_are_exact_over_the_exponent_range(span):
    """Values over 2^span in one column, infinities in another problem: the centroids are the
    exact integers' (rounded at 2^-94 of the column's largest value), whatever the path."""
    rng = np.random.default_rng(span)
    n, d, k = 3000, 5, 4
    X = (rng.choice([-1.0, 1.0], (n, d)) * 2.0 ** rng.uniform(-span, 0, (n, d))).astype(np.float32)
    X[0] = 1.0
    C0 = X[:k].copy()
    desc = kmeans.descriptor(np.float32).set_cluster_count(k).set_max_iteration_count(1)
    desc.set_compute_form(kmeans.compute_form.plain)
    r = kmeans.train(desc, X, C0)
    lab = kmeans.infer(desc, kmeans.model(C0), X).get_responses().ravel()
    from fractions import Fraction
    for j in range(k):
        rows = X[lab == j]
        if len(rows) < 2:
            continue
        for t in range(d):
            unit = Fraction(2) ** (int(np.frexp(np.abs(X[:, t]).max())[1]) - 94)
            total = sum(round(Fraction(float(v)) / unit) for v in rows[:, t]) * unit
            s = float(total)  # the nearest double
            want = np.float32(s / len(rows))
            assert r.get_model().get_centroids()[j, t] == want, (j, t)


def test_infinite_rows_take_the_same_sums_as_the_general_path():
    rng = np.random.default_rng(5)
    X = rng.standard_normal((2000, 6)).astype(np.float32)
    X[7, 2] = np.inf
    X[1500, 0] = np.nan
    desc = kmeans.descriptor(np.float32).set_cluster_count(5).set_max_iteration_count(2)
    desc.set_compute_form(kmeans.compute_form.plain)
    a = kmeans.train(desc, X, X[10:15].copy())
    b = kmeans.train(desc.set_recheck(True), X, X[10:15].copy())
    np.testing.assert_array_equal(a.get_model().get_centroids(), b.get_model().get_centroids())


def _train_args(n=5000, d=20, k=20, T=4):
    X, C0 = _data(n, d, k, np.float32, 7, False)
    desc = kmeans.descriptor(np.float32).set_cluster_count(k).set_max_iteration_count(T)
    return desc.set_compute_form(kmeans.compute_form.plain), torch.from_numpy(X).cuda(), torch.from_numpy(C0).cuda()


def test_kernel_times_are_still_told_apart():
    """With kernel timing on, a train's assignments and updates are timed one by one."""
    ctx = _native.context(0)
    args = _train_args()
    alone = kmeans.train(*args)
    ctx.check(ctx.lib.kmb_context_set_kernel_timing(ctx.handle, 1))
    try:
        timed = kmeans.train(*args)
        ms, launches = ctypes.c_double(), ctypes.c_int64()
        counts = {}
        for kernel in (0, 2):
            ctx.check(ctx.lib.kmb_context_kernel_time(ctx.handle, kernel, ctypes.byref(ms), ctypes.byref(launches)))
            counts[kernel] = launches.value
            assert ms.value > 0
    finally:
        ctx.check(ctx.lib.kmb_context_set_kernel_timing(ctx.handle, 0))
    assert counts == {0: 5, 2: 4}
    assert torch.equal(alone.get_model().get_centroids(), timed.get_model().get_centroids())
    assert torch.equal(alone.get_responses(), timed.get_responses())


def test_a_train_without_recheck_leaves_no_rechecked_rows():
    """kmb_context_recheck_rows is about the context's last pass, not an earlier call's."""
    ctx = _native.context(0)
    desc, X, C = _train_args()
    tied = torch.cat([C, C])  # every row's two nearest clusters tie
    tc = kmeans.descriptor(np.float32).set_cluster_count(40).set_compute_form(kmeans.compute_form.bf16x3)
    kmeans.infer(tc, kmeans.model(tied), X)
    count = ctypes.c_int64()
    ctx.check(ctx.lib.kmb_context_recheck_rows(ctx.handle, None, 0, ctypes.byref(count)))
    assert count.value == X.shape[0]
    kmeans.train(desc, X, C)
    ctx.check(ctx.lib.kmb_context_recheck_rows(ctx.handle, None, 0, ctypes.byref(count)))
    assert count.value == 0


def test_grid_stays_within_the_contexts_sms(tmp_path):
    """kmb_context_set_max_sms bounds the grid of this persistent launch too."""
    from torch.profiler import ProfilerActivity, profile
    ctx = _native.context(0)
    args = _train_args()
    alone = kmeans.train(*args)
    ctx.check(ctx.lib.kmb_context_set_max_sms(ctx.handle, 3))
    try:
        with profile(activities=[ProfilerActivity.CUDA]) as p:
            few = kmeans.train(*args)
            torch.cuda.synchronize()
    finally:
        ctx.check(ctx.lib.kmb_context_set_max_sms(ctx.handle, 0))
    p.export_chrome_trace(str(tmp_path / "trace.json"))
    events = json.load(open(tmp_path / "trace.json"))["traceEvents"]
    grids = [e["args"]["grid"][0] for e in events if "small_train_kernel" in e.get("name", "")]
    assert grids and max(grids) <= 3, grids
    assert torch.equal(alone.get_model().get_centroids(), few.get_model().get_centroids())
