"""Row-streaming kernels at the edges of their load widths: rows of 16-, 8- and 4-byte
multiples at aligned and shifted bases, narrow and wide, one row and ragged blocks --
objective and tensor-core responses against the FP64 evaluation, k-means++ rows against the
oracle."""
import numpy as np
import pytest
import torch

from onedal_b200 import kmeans
from oracle import restated

pytestmark = pytest.mark.gpu


def _shifted(X, shift):
    """A contiguous CUDA copy of X whose base is `shift` elements past an aligned one."""
    buf = torch.zeros(X.size + shift, dtype=torch.from_numpy(X).dtype, device="cuda")
    buf[shift:] = torch.from_numpy(X).cuda().reshape(-1)
    return buf[shift:].view(*X.shape)


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("n,d,k", [(1, 1, 1), (3, 2, 2), (1185, 5, 3), (5000, 50, 7), (4999, 64, 9), (700, 130, 5),
                                   (300, 256, 4), (70, 513, 3)])
@pytest.mark.parametrize("shift", [0, 1, 2])
def test_objective_and_responses(dt, n, d, k, shift):
    rng = np.random.default_rng(n + d)
    X = rng.standard_normal((n, d)).astype(dt)
    C = rng.standard_normal((k, d)).astype(dt)
    want, obj = restated.infer(X.astype(np.float64), C.astype(np.float64), True)
    forms = [kmeans.compute_form.plain]
    if dt == np.float32 and d <= 256:
        forms.append(kmeans.compute_form.bf16x3)
    for form in forms:
        desc = kmeans.descriptor(dt).set_cluster_count(k).set_compute_form(form)
        desc.set_result_options(kmeans.result_options.compute_exact_objective_function)
        r = kmeans.infer(desc, kmeans.model(_shifted(C, shift)), _shifted(X, shift))
        got = r.get_responses().cpu().numpy().ravel()
        assert (got == want).mean() > 0.999 if form == kmeans.compute_form.plain else (got == want).all()
        # both FP64 sums of n * d squares: relative 2 n d 2^-53; responses that differ by a near tie move less
        assert abs(r.get_objective_function_value() - obj) <= 1e-6 * obj
        if (got == want).all():
            assert abs(r.get_objective_function_value() - obj) <= 4 * n * d * 2.0 ** -53 * obj


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("n,d", [(40, 1), (511, 3), (513, 7), (3000, 20), (2049, 50), (1025, 69), (1100, 70), (600, 131)])
def test_plusplus_rows(dt, n, d):
    rng = np.random.default_rng(d)
    X = rng.standard_normal((n, d)).astype(dt)
    got = kmeans.init_plusplus(torch.from_numpy(X).cuda(), 12, dt).cpu().numpy()
    np.testing.assert_array_equal(got, restated.init_plusplus(X, 12)[0])
