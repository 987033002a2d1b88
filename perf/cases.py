"""The k-means work that is timed: train, infer, CSR rows, the default initialisation and the
batched form, each through the package's public calls.

A case is a dict of plain values:

    kind        train | train_init | infer | train_csr | batched
    data        how the rows are drawn: blobs | anisotropic | bisector | serving | sparse
    n, d, k     rows, columns, clusters (batched: n problems, each with sizes of its own)
    dtype       float32 | float64
    iterations  the descriptor's max_iteration_count (accuracy_threshold stays at its default, 0)
    form        auto (the descriptor's default) | plain
    objective   infer: whether the exact objective is asked for

Rows and centroids are CUDA tensors, as a program that keeps its data on the GPU has them.
"""
import numpy as np
import torch

from onedal_b200 import kmeans, workloads
from onedal_b200.batched import batched_train

DEVICE = "cuda"
CSR_ENTRIES = 64  # stored entries per sparse row


def _case(name, kind, data, n, d, k, dtype="float32", iterations=0, form="auto", objective=False):
    return {"name": name, "kind": kind, "data": data, "n": n, "d": d, "k": k, "dtype": dtype,
            "iterations": iterations, "form": form, "objective": objective}


def listed():
    return [
        # The smallest train a program makes: the size of the reference's known-answer test, doubles
        # (what numpy holds by default), to convergence. Launches and latency.
        _case("train_tiny_f64", "train", "blobs", 100, 3, 3, "float64", 100),
        # One infer request against a resident model: the median request of the serving workload,
        # with a ragged row and cluster count.
        _case("infer_request_f32", "infer", "serving", 4097, 64, 300),
        # The reference's example-sized training set, 20 blobs, in both float types.
        _case("train_blobs_f32", "train", "blobs", 100_000, 20, 20, "float32", 50),
        _case("train_blobs_f64", "train", "blobs", 100_000, 20, 20, "float64", 50),
        # An ordinary double-precision train at odd sizes (rows of 37 columns, not 16-byte multiples).
        _case("train_ragged_f64", "train", "blobs", 300_007, 37, 101, "float64", 15),
        # The call without initial centroids (k-means++), few clusters, 50 columns, three million rows.
        _case("train_default_f32", "train_init", "blobs", 3_000_000, 50, 20, "float32", 10),
        # Many clusters for narrow rows: a million rows of 20 columns, 1000 clusters.
        _case("train_narrow_f32", "train", "blobs", 1_000_000, 20, 1000, "float32", 10),
        # FP32 training at scale with the plain form asked for.
        _case("train_plain_f32", "train", "anisotropic", 10_000_000, 64, 256, "float32", 10, "plain"),
        # The headline: 20M x 128, 1024 clusters, a tenth of the rows near ties, 20 iterations.
        _case("train_large_f32", "train", "bisector", 20_000_000, 128, 1024, "float32", 20),
        # Labelling a large table against a fitted model, with the objective.
        _case("infer_large_f32", "infer", "bisector", 4_000_001, 128, 1024, objective=True),
        # Sparse rows (method::lloyd_csr): text-like width, 64 entries a row.
        _case("train_csr_f32", "train_csr", "sparse", 500_000, 20_000, 256, "float32", 10),
        # Many independent problems in one call (1,000..200,000 rows, 8..64 columns, 4..128 clusters each).
        _case("batched_f32", "batched", "blobs", 512, 64, 128, "float32", 30),
    ]


def _log_int(rng, lo, hi):
    return int(round(float(np.exp(rng.uniform(np.log(lo), np.log(hi))))))


def draw(rng):
    kind = rng.choice(["train", "train", "train", "train", "infer", "infer", "train_init", "train_csr", "batched"])
    dtype = "float64" if kind in ("train", "infer") and rng.random() < 0.35 else "float32"
    if kind == "batched":
        return _unnamed(_case("", kind, "blobs", _log_int(rng, 3, 500), 64, 128, iterations=rng.randint(5, 30)))
    if kind == "train_csr":
        n, k = _log_int(rng, 2_000, 500_000), _log_int(rng, 5, 256)
        return _unnamed(_case("", kind, "sparse", n, _log_int(rng, 1_000, 20_000), k, iterations=rng.randint(3, 10)))
    d = rng.choice([20, 32, 50, 64, 84, 128, 0, 0, 0, 0, 0, 0]) or _log_int(rng, 3, 130)
    k = _log_int(rng, 3, 200 if kind == "train_init" else 1024)
    n = _log_int(rng, max(100, 4 * k), 3_000_000 if kind == "train_init" else 20_000_000)
    passes = 0 if kind == "infer" else rng.randint(5, 50)
    form = "plain" if dtype == "float32" and kind != "train_init" and rng.random() < 0.2 else "auto"
    # no more than the largest listed case, by the rate of the arithmetic that the case takes
    flops = 1.5e12 if dtype == "float64" else (4e12 if form == "plain" else 3e13)
    n = int(max(4 * k, min(n, flops / (2.0 * k * max(d, 16) * (passes + 1)), 1.5e9 / d)))
    data = rng.choice(["blobs", "anisotropic", "bisector"]) if kind != "infer" else rng.choice(["serving", "blobs", "bisector"])
    return _unnamed(_case("", kind, data, n, d, k, dtype, passes, form, kind == "infer" and rng.random() < 0.5))


def _unnamed(case):
    return {key: v for key, v in case.items() if key != "name"}


def _dtype(case):
    return torch.float64 if case["dtype"] == "float64" else torch.float32


def _rows(data, n, d, k, seed, dtype):
    """(rows, the centres they were drawn around)."""
    if data == "anisotropic":
        return workloads.anisotropic_blobs(n, d, k, seed, DEVICE, dtype=dtype)
    if data == "bisector":
        return workloads.bisector_blobs(n, d, k, seed, DEVICE, dtype=dtype)
    return workloads.blobs(n, d, k, seed, DEVICE, dtype=dtype)


def _descriptor(case):
    method = kmeans.method.lloyd_csr if case["kind"] == "train_csr" else kmeans.method.lloyd_dense
    desc = kmeans.descriptor(np.dtype(case["dtype"]), method).set_cluster_count(case["k"])
    desc.set_max_iteration_count(case["iterations"])
    if case["form"] == "plain":
        desc.set_compute_form(kmeans.compute_form.plain)
    if case["objective"]:
        desc.set_result_options(kmeans.result_options.compute_exact_objective_function)
    return desc


def _spread_rows(X, k):
    """k distinct rows (the rows are drawn independently, so any will do), as initial centroids."""
    return X[torch.arange(k, device=X.device) * (X.shape[0] // k)].clone()


def _sparse(n, d, seed):
    """One entry per column stripe: values N(0, 1), int64 indices, zero-based."""
    g = torch.Generator(device=DEVICE)
    g.manual_seed(seed)
    per = CSR_ENTRIES
    stripe = d // per
    cols = torch.randint(0, stripe, (n, per), device=DEVICE, generator=g) + torch.arange(per, device=DEVICE) * stripe
    vals = torch.randn(n, per, device=DEVICE, generator=g)
    offs = torch.arange(0, n * per + 1, per, device=DEVICE)
    return vals, cols, offs


def _problems(case, seed):
    rng = np.random.default_rng(1004)  # the problems' sizes; their values come from the seed
    g = torch.Generator(device=DEVICE)
    g.manual_seed(seed)
    out = []
    for _ in range(case["n"]):
        n = int(np.exp(rng.uniform(np.log(1e3), np.log(2e5))))
        d = int(rng.choice([8, 16, 32, 64]))
        k = int(round(np.exp(rng.uniform(np.log(4), np.log(128)))))
        centres = torch.rand(k, d, generator=g, device=DEVICE) * 20 - 10
        lab = torch.randint(0, k, (n,), generator=g, device=DEVICE)
        X = centres[lab] + torch.randn(n, d, generator=g, device=DEVICE)
        out.append((X, _spread_rows(X, k)))
    return out


def prepare(case, seed):
    n, d, k, kind = case["n"], case["d"], case["k"], case["kind"]
    state = {"case": case, "desc": _descriptor(case)}
    if kind == "batched":
        state["problems"] = _problems(case, seed)
    elif kind == "train_csr":
        vals, cols, offs = _sparse(n, d, seed)
        state["X"] = kmeans.csr_table(vals.reshape(-1), cols.reshape(-1), offs, n, d, kmeans.sparse_indexing.zero_based)
        pick = torch.arange(k, device=DEVICE) * (n // k)
        state["C"] = torch.zeros(k, d, device=DEVICE).scatter_(1, cols[pick], vals[pick])
    elif case["data"] == "serving":  # a resident model and one request's rows
        g = torch.Generator(device=DEVICE)
        g.manual_seed(seed)
        state["X"] = torch.randn(n, d, generator=g, device=DEVICE, dtype=_dtype(case))
        state["C"] = torch.rand(k, d, generator=g, device=DEVICE, dtype=_dtype(case)) * 2 - 1
    else:
        X, centres = _rows(case["data"], n, d, k, seed, _dtype(case))
        state["X"] = X
        # infer: a fitted model of these rows; train: k of the rows to start from
        state["C"] = centres.to(_dtype(case)) if kind == "infer" else _spread_rows(X, k)
    if kind == "infer":
        state["model"] = kmeans.model(state["C"])
    return state


def run(state):
    kind, desc = state["case"]["kind"], state["desc"]
    if kind == "batched":
        results, _ = batched_train(state["problems"], state["case"]["iterations"])
        return {"centroids": torch.cat([c.reshape(-1) for c, _, _ in results]),
                "responses": torch.cat([r for _, r, _ in results]),
                "iterations": torch.tensor([i for _, _, i in results])}
    if kind == "infer":
        r = kmeans.infer(desc, state["model"], state["X"])
        out = {"responses": r.get_responses()}
        if state["case"]["objective"]:
            out["objective"] = r.get_objective_function_value()
        return out
    r = kmeans.train(desc, state["X"]) if kind == "train_init" else kmeans.train(desc, state["X"], state["C"])
    return {"centroids": r.get_model().get_centroids(), "responses": r.get_responses(),
            "iterations": r.get_iteration_count(), "objective": r.get_objective_function_value()}


def work(case):
    """Rows, initial centroids in; centroids and labels out; 2nkd operations per assignment."""
    n, d, k, kind = case["n"], case["d"], case["k"], case["kind"]
    size = 8 if case["dtype"] == "float64" else 4
    if kind == "batched":  # means of the problems' distributions (n about 37,600, d 30, k 36)
        rows, cols, clusters = 37_600.0 * n, 30.0, 36.0
        return {"bytes": rows * (4 * cols + 4), "flops": 2 * rows * cols * clusters * case["iterations"]}
    if kind == "train_csr":
        nnz = float(n) * CSR_ENTRIES
        return {"bytes": nnz * 12 + n * 12 + 8.0 * k * d, "flops": 2 * nnz * k * (case["iterations"] + 1)}
    flops = 2.0 * n * d * k * (case["iterations"] + 1)
    if kind == "train_init":
        flops += 3.0 * n * d * (k - 1)  # one distance to every new center
    return {"bytes": float(size) * (n * d + 2 * k * d) + 4.0 * n, "flops": flops}


# ---- the same in 64 bits ----------------------------------------------------------

def _assign64(X, C):
    """Labels and squared distances of the rows, in row blocks."""
    h = 0.5 * (C * C).sum(1)
    step = max(1, int(2.5e8 // C.shape[0]))
    labels, dist = [], []
    for s in range(0, X.shape[0], step):
        x = X[s:s + step].double()
        best, lab = (h - x @ C.T).min(1)
        labels.append(lab)
        dist.append(2 * best + (x * x).sum(1))
    return torch.cat(labels), torch.cat(dist)


def _sums64(X, labels, k):
    step = max(1, int(2.5e8 // k))
    sums = torch.zeros(k, X.shape[1], dtype=torch.float64, device=X.device)
    for s in range(0, X.shape[0], step):
        one_hot = torch.nn.functional.one_hot(labels[s:s + step], k).double()
        sums += one_hot.T @ X[s:s + step].double()
    return sums, torch.bincount(labels, minlength=k)


def _objective64(X, C, labels):
    step = 1 << 21
    return float(sum(((X[s:s + step].double() - C[labels[s:s + step]]) ** 2).sum() for s in range(0, X.shape[0], step)))


def _lloyd64(X, C, iterations):
    C, done = C.double(), 0
    k = C.shape[0]
    for _ in range(iterations):
        labels, dist = _assign64(X, C)
        sums, counts = _sums64(X, labels, k)
        new = sums / counts.clamp(min=1).unsqueeze(1)
        empty = torch.nonzero(counts == 0).reshape(-1)
        if len(empty):
            new[empty] = X[torch.topk(dist, len(empty)).indices].double()
        done += 1
        still = bool((new == C).all())
        C = new
        if still:
            break
    return C, done


def exact(case, seed):
    kind = case["kind"]
    if work(case)["flops"] > 1e13 or (kind == "infer" and not case["objective"]):
        return None  # too long, or whole numbers alone
    if kind == "train_init":  # which rows k-means++ draws is decided in the data's own type
        return None
    state = prepare(case, seed)
    if kind == "batched":
        return {"centroids": torch.cat([_lloyd64(X, C, case["iterations"])[0].reshape(-1) for X, C in state["problems"]]),
                "responses": None, "iterations": None}
    X, C = state["X"], state["C"]
    if kind == "train_csr":
        return _exact_csr(case, X, C)
    if kind == "infer":
        C = C.double()
        return {"responses": None, "objective": _objective64(X, C, _assign64(X, C)[0])}
    C, _ = _lloyd64(X, C, case["iterations"])
    return {"centroids": C, "responses": None, "iterations": None, "objective": _objective64(X, C, _assign64(X, C)[0])}


def _exact_csr(case, table, C):
    n, d, k = case["n"], case["d"], case["k"]
    vals, cols = table.data.double().reshape(n, -1), table.column_indices.reshape(n, -1)
    sparse = torch.sparse_csr_tensor(table.row_offsets, cols.reshape(-1), vals.reshape(-1), (n, d))
    C = C.double()

    def assign(C):
        s = 0.5 * (C * C).sum(1) - sparse @ C.T.contiguous()
        best, lab = s.min(1)
        return lab, 2 * best + (vals * vals).sum(1)

    for _ in range(case["iterations"]):
        lab, dist = assign(C)
        at = (lab.unsqueeze(1) * d + cols).reshape(-1)
        sums = torch.zeros(k * d, dtype=torch.float64, device=C.device).index_add_(0, at, vals.reshape(-1)).reshape(k, d)
        counts = torch.bincount(lab, minlength=k)
        new = sums / counts.clamp(min=1).unsqueeze(1)
        for j, row in zip(torch.nonzero(counts == 0).reshape(-1).tolist(), torch.topk(dist, int((counts == 0).sum())).indices):
            new[j] = torch.zeros(d, dtype=torch.float64, device=C.device).scatter_(0, cols[row], vals[row])
        still = bool((new == C).all())
        C = new
        if still:
            break
    return {"centroids": C, "responses": None, "iterations": None, "objective": float(assign(C)[1].clamp(min=0).sum())}
