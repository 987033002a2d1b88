"""Calls from several host threads, a context each: every call's result is the one that it
gives alone. Each pair of jobs reaches one kernel with different amounts of dynamic shared
memory, whose limit is an attribute that the threads share. And no thread's small train waits
for another's long one."""
import threading
import time

import numpy as np
import pytest
import torch

from onedal_b200 import kmeans
from onedal_b200.batched import batched_train

pytestmark = pytest.mark.gpu


def _rows(n, d, k, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed + n + d + k)
    c = torch.rand(k, d, device="cuda", generator=g) * 20 - 10
    X = c[torch.randint(0, k, (n,), device="cuda", generator=g)] + torch.randn(n, d, device="cuda", generator=g)
    return X, X[:: n // k][:k].contiguous()


def _init(n, d, k):
    X, _ = _rows(n, d, k)
    return lambda: [kmeans.init_plusplus(X, k, np.float32)]


def _infer(n, d, k, form):
    X, C = _rows(n, d, k)
    desc = kmeans.descriptor(np.float32).set_cluster_count(k).set_compute_form(form)
    return lambda: [kmeans.infer(desc, kmeans.model(C), X).get_responses()]


def _train(n, d, k):
    X, C = _rows(n, d, k)
    desc = kmeans.descriptor(np.float32).set_cluster_count(k).set_max_iteration_count(5)
    desc.set_compute_form(kmeans.compute_form.plain)

    def job():
        r = kmeans.train(desc, X, C)
        return [r.get_responses(), r.get_model().get_centroids()]
    return job


def _csr(n, d, k, per_row=8):
    g = torch.Generator(device="cuda").manual_seed(d)
    cols = torch.sort(torch.rand(n, d, device="cuda", generator=g).topk(per_row, dim=1).indices, dim=1).values
    vals = torch.randn(n, per_row, device="cuda", generator=g)
    offs = torch.arange(0, n * per_row + 1, per_row, device="cuda")
    X = kmeans.csr_table(vals.reshape(-1), cols.reshape(-1), offs, n, d, kmeans.sparse_indexing.zero_based)
    C = torch.zeros(k, d, device="cuda").scatter_(1, cols[:k], vals[:k])
    desc = kmeans.descriptor(np.float32, kmeans.method.lloyd_csr).set_cluster_count(k).set_max_iteration_count(2)

    def job():
        r = kmeans.train(desc, X, C)
        return [r.get_responses(), r.get_model().get_centroids()]
    return job


def _batched(n, d, k):
    problems = [_rows(n, d, k, s) for s in range(4)]
    return lambda: [t for c, r, _ in batched_train(problems, 4)[0] for t in (c, r)]


def _host(values):
    torch.cuda.current_stream().synchronize()
    return [v.cpu().numpy() if isinstance(v, torch.Tensor) else np.asarray(v) for v in values]


PLAIN, TC = kmeans.compute_form.plain, kmeans.compute_form.bf16x3


@pytest.mark.parametrize("make", [
    pytest.param(lambda: (_init(200_000, 50, 60), _init(200_000, 10, 60)), id="init"),
    pytest.param(lambda: (_infer(20_000, 100, 200, TC), _infer(20_000, 30, 200, TC)), id="one_cluster_tile"),
    pytest.param(lambda: (_infer(20_000, 250, 600, TC), _infer(20_000, 30, 600, TC)), id="cluster_tiles"),
    pytest.param(lambda: (_infer(1 << 18, 64, 512, PLAIN), _infer(1 << 18, 64, 256, PLAIN)), id="resident"),
    pytest.param(lambda: (_train(30_000, 60, 30), _train(3_000, 60, 30)), id="small"),
    pytest.param(lambda: (_csr(2_000, 20_000, 20), _csr(2_000, 2_000, 20)), id="csr"),
    pytest.param(lambda: (_batched(3_000, 60, 200), _batched(3_000, 5, 6)), id="batched"),
])
def test_threads_get_what_they_get_alone(make):
    jobs = make()
    want = [_host(job()) for job in jobs]
    torch.cuda.synchronize()
    wrong, gate = [], threading.Barrier(len(jobs))

    def work(i):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(40):
                    gate.wait(60)
                    got = _host(jobs[i]())
                    if not all(np.array_equal(a, b) for a, b in zip(got, want[i])):
                        wrong.append(f"job {i}: other results")
        except Exception as e:  # a refused launch
            wrong.append(f"job {i}: {e}")
            gate.abort()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong[:3]


@pytest.mark.parametrize("n", [100, 2000], ids=["one_block", "blocks"])
def test_a_small_train_does_not_wait_for_another_threads(n):
    """A train of eight blocks that never converges (a NaN in doubles makes every shift a NaN)
    runs for its 25,000 iterations; a thread with a few blocks' train, which the other SMs can
    hold, is done long before."""
    def args(n, T):
        X, C = (t.double() for t in _rows(n, 20, 20))
        return kmeans.descriptor(np.float64).set_cluster_count(20).set_max_iteration_count(T), X, C
    long_args, short_args = args(2001, 25_000), args(n, 3)
    long_args[1][5, 5] = float("nan")
    kmeans.train(*short_args)
    ended = {}

    def work(name, a):
        with torch.cuda.stream(torch.cuda.Stream()):
            kmeans.train(*a)
        ended[name] = time.perf_counter()

    threads = [threading.Thread(target=work, args=("long", long_args)), threading.Thread(target=work, args=("short", short_args))]
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    threads[0].start()
    time.sleep(0.03)
    threads[1].start()
    for t in threads:
        t.join()
    assert ended["long"] - t0 > 0.15, "the long train was over before the other began"
    assert ended["long"] - ended["short"] > 0.05, ended
