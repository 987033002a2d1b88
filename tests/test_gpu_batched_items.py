"""Batched problems with few rows per work item (few problems: 512-row items, handed out one
by one) give each problem's single-problem result bit for bit: items of one row, full and
ragged ones, one problem and several."""
import ctypes

import numpy as np
import pytest
import torch

from onedal_b200 import _native
from onedal_b200.batched import batched_train

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[(511, 3, 4)], [(512, 64, 128)], [(513, 8, 5)], [(70_001, 32, 33)],
                                   [(1, 1, 1), (1025, 17, 200), (40_000, 64, 100), (3000, 24, 16)]])
def test_few_problems_equal_single_ones(sizes):
    rng = np.random.default_rng(len(sizes) + sizes[0][0])
    problems = []
    for n, d, k in sizes:
        c = rng.uniform(-10, 10, (k, d))
        X = (c[rng.integers(0, k, n)] + rng.standard_normal((n, d))).astype(np.float32)
        problems.append((torch.from_numpy(X).cuda(), torch.from_numpy(X[rng.permutation(n)[:k]].copy()).cuda()))
    results, _ = batched_train(problems, 12)
    ctx = _native.context(0)
    ctx.set_stream(torch.cuda.current_stream().cuda_stream)
    for (X, C0), (C, lab, iters) in zip(problems, results):
        n, d, k = X.shape[0], X.shape[1], C0.shape[0]
        one, labels, it = C0.clone(), torch.empty(n, dtype=torch.int32, device="cuda"), ctypes.c_int64()
        p = _native.kmb_params(k, 12, 0.0, _native.KMB_FORM_PLAIN, 0)
        ctx.check(ctx.lib.kmb_lloyd_iterate(ctx.handle, _native.KMB_F32, X.data_ptr(), n, d, one.data_ptr(),
                                            ctypes.byref(p), labels.data_ptr(), ctypes.byref(it), None))
        assert it.value == iters
        assert torch.equal(one, C) and torch.equal(labels, lab)
