"""The workloads whose speed this framework is judged by, each through its
public entry points.

``listed()`` names them; ``draw(rng)`` gives another one of the same ranges;
``prepare`` makes a case's inputs (from the seed alone) and the trees or plans
a user's program keeps; ``run`` is one pass; ``work`` says what a pass cannot
do without; ``exact`` gives the outputs in 64-bit arithmetic where plain torch
can compute them in reasonable time.

The operations ("op"):

* query:   ``tree.query`` on a tree that was built before;
* rebuild: ``build_kd_tree`` and a query of it, as programs do whose cloud
  changes from frame to frame;
* grad:    a query with gradients for both clouds and its backward pass;
* batch:   ``BatchedKDTrees.query_flat``, many clouds with a tree and a k each
  and their queries in one tensor;
* chamfer: ``nn_distance_bidirectional`` and its backward pass (the training
  loss this operator is known for);
* brute:   ``nn_distance``, the exhaustive search, in one of its modes.
"""
import math

import numpy as np
import torch

from torch_kdtree_gb300 import build_kd_tree, nn_distance, nn_distance_bidirectional
from torch_kdtree_gb300.batched import BatchedKDTrees

DEVICE = "cuda"
DTYPES = {"float32": torch.float32, "float64": torch.float64}


def listed():
    return [
        # A handful of neighbours in a small cloud (a mesh, a molecule): latency only.
        {"name": "query_small", "op": "query", "n": 1000, "nq": 200, "k": 10, "d": 3, "dtype": "float32",
         "cloud": "normal", "scale": 1.0},
        # The plain benchmark configuration: one scan's points looked up in a model cloud.
        {"name": "query_plain", "op": "query", "n": 100_000, "nq": 10_000, "k": 5, "d": 3, "dtype": "float32",
         "cloud": "normal", "scale": 1e3},
        # The headline cloud (volume and surface points, queries partly outside) at default options.
        {"name": "query_large", "op": "query", "n": 4_194_304, "nq": 1_048_576, "k": 16, "d": 3, "dtype": "float32",
         "cloud": "cube_sphere", "scale": 1.0},
        # The published benchmark setting's largest k: density estimation, normals from wide neighbourhoods.
        {"name": "query_k100", "op": "query", "n": 1_000_000, "nq": 1_000_000, "k": 100, "d": 3, "dtype": "float32",
         "cloud": "normal", "scale": 1e3},
        # Double precision: survey and simulation coordinates.
        {"name": "query_double", "op": "query", "n": 200_000, "nq": 65_536, "k": 8, "d": 3, "dtype": "float64",
         "cloud": "normal", "scale": 1.0},
        # Feature vectors in a tree of more than three dimensions.
        {"name": "query_6d", "op": "query", "n": 1_000_000, "nq": 65_536, "k": 16, "d": 6, "dtype": "float32",
         "cloud": "normal", "scale": 1.0},
        # A cloud that is new every time (registration, simulation steps): build, then query.
        {"name": "rebuild_1m", "op": "rebuild", "n": 1_048_576, "nq": 65_536, "k": 8, "d": 3, "dtype": "float32",
         "cloud": "normal", "scale": 1.0},
        # The differentiable configuration: both clouds take gradients.
        {"name": "grad_1m", "op": "grad", "n": 1_048_576, "nq": 1_048_576, "k": 8, "d": 3, "dtype": "float32",
         "cloud": "normal", "scale": 1.0},
        # The batched configuration: 256 ragged clouds, k of 1, 4 or 16 per cloud.
        {"name": "batch_256", "op": "batch", "clouds": 256, "lo": 1000, "hi": 200_000, "sizes": 0, "d": 3,
         "dtype": "float32"},
        # The two-way nearest-neighbour loss between two clouds, with gradients.
        {"name": "chamfer_64k", "op": "chamfer", "n": 65_536, "nq": 65_536, "k": 1, "d": 3, "dtype": "float32"},
        # The exhaustive configuration at default options: exact neighbours of embeddings.
        {"name": "brute_exact_32d", "op": "brute", "n": 262_144, "nq": 65_536, "k": 32, "d": 32, "dtype": "float32",
         "mode": "exact"},
        # The same search through the tensor cores (the same answer).
        {"name": "brute_tf32_32d", "op": "brute", "n": 262_144, "nq": 65_536, "k": 32, "d": 32, "dtype": "float32",
         "mode": "tf32"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["query", "query", "rebuild", "grad", "batch", "chamfer", "brute"])
    if op == "query":
        d = rng.choice([1, 2, 3, 3, 3, 4, 5, 6, 8])
        wide = d > 3
        double = rng.random() < 0.2
        n = _log_int(rng, 1000, 1_000_000 if wide or double else 4_194_304)
        nq = _log_int(rng, 200, 65_536 if wide or double else 1_048_576)
        k = rng.choice([1, 4, 5, 8, 10, 16] if wide or double else [1, 4, 5, 8, 10, 16, 20, 33, 100])
        cloud = "cube_sphere" if d == 3 and rng.random() < 0.4 else "normal"
        case = {"op": op, "n": n, "nq": nq, "k": k, "d": d, "dtype": "float64" if double else "float32",
                "cloud": cloud, "scale": rng.choice([1.0, 1e3])}
        if rng.random() < 0.25:  # a depth of the caller's choice: 8 to 64 points per leaf
            case["levels"] = max(1, int(math.log2(n)) - rng.randint(3, 6))
        return case
    if op == "rebuild":
        return {"op": op, "n": _log_int(rng, 1000, 4_194_304), "nq": _log_int(rng, 200, 262_144),
                "k": rng.choice([1, 8, 16]), "d": rng.choice([2, 3, 3, 6]),
                "dtype": "float64" if rng.random() < 0.15 else "float32", "cloud": "normal", "scale": 1.0}
    if op == "grad":
        return {"op": op, "n": _log_int(rng, 1000, 1_048_576), "nq": _log_int(rng, 1000, 1_048_576),
                "k": rng.choice([1, 4, 8, 16]), "d": rng.choice([2, 3, 3]), "dtype": "float32", "cloud": "normal",
                "scale": 1.0}
    if op == "batch":
        return {"op": op, "clouds": _log_int(rng, 4, 256), "lo": 1000, "hi": _log_int(rng, 2000, 200_000),
                "sizes": rng.randint(1, 1 << 30), "d": 3, "dtype": "float32"}
    if op == "chamfer":
        return {"op": op, "n": _log_int(rng, 500, 65_536), "nq": _log_int(rng, 500, 65_536), "k": 1,
                "d": rng.choice([2, 3, 3]), "dtype": "float32"}
    return {"op": op, "n": _log_int(rng, 1000, 262_144), "nq": _log_int(rng, 128, 65_536),
            "k": rng.choice([1, 8, 16, 32]), "d": rng.choice([3, 8, 8, 13, 16, 32, 32]), "dtype": "float32",
            "mode": rng.choice(["exact", "exact", "tf32", "bf16_split"])}


# ---------------------------------------------------------------- inputs --

def _normal(gen, rows, d, dtype):
    return torch.randn(rows, d, generator=gen, device=DEVICE, dtype=dtype)


def _uniform(gen, rows, d, dtype):
    return torch.rand(rows, d, generator=gen, device=DEVICE, dtype=dtype)


def _clouds(case, gen):
    """(references, queries) of one case."""
    n, nq, d, dtype = case["n"], case["nq"], case["d"], DTYPES[case["dtype"]]
    if case.get("cloud") == "cube_sphere":
        # half the points uniform in the unit cube, half on a sphere around its centre with radial noise;
        # queries uniform in a slightly larger cube
        h = n // 2
        dirs = _normal(gen, n - h, 3, dtype)
        dirs /= dirs.norm(dim=1, keepdim=True)
        radius = 1.0 + 0.01 * _normal(gen, n - h, 1, dtype)
        ref = torch.cat([_uniform(gen, h, 3, dtype), 0.5 + radius * dirs])
        q = _uniform(gen, nq, 3, dtype) * 1.2 - 0.1
    else:
        ref = _normal(gen, n, d, dtype)
        q = _normal(gen, nq, d, dtype)
    if case["op"] == "brute":
        # 5% of the references are exact copies of others, as embeddings of repeated items are
        m = n // 20
        perm = torch.randperm(n, generator=gen, device=DEVICE)
        ref[perm[:m]] = ref[perm[m:2 * m]]
    scale = case.get("scale", 1.0)
    return (ref * scale, q * scale) if scale != 1.0 else (ref, q)


def _batch_plan(case):
    """Sizes, query counts and k of every cloud: part of the case, not of the seed."""
    rng = np.random.default_rng(case["sizes"])
    n = np.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"]), case["clouds"])).round().astype(int)
    ks = rng.choice([1, 4, 16], case["clouds"])
    return [int(v) for v in n], [int(v) // 2 for v in n], [int(v) for v in ks]


def _mixture(gen, rows, means, sigma, dtype):
    comp = torch.randint(0, means.shape[0], (rows,), generator=gen, device=DEVICE)
    return means[comp] + _normal(gen, rows, means.shape[1], dtype) * sigma[comp]


def _batch_clouds(case, gen):
    d, dtype = case["d"], DTYPES[case["dtype"]]
    refs, qs = [], []
    sizes, counts, _ = _batch_plan(case)
    for n, nq in zip(sizes, counts):
        means = _uniform(gen, 8, d, dtype) * 20.0 - 10.0
        sigma = _uniform(gen, 8, 1, dtype) * 1.9 + 0.1
        refs.append(_mixture(gen, n, means, sigma, dtype))
        qs.append(_mixture(gen, nq, means, sigma, dtype))
    return refs, qs


def _inputs(case, seed):
    """Every input tensor of a case, from the seed alone."""
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(seed)
    if case["op"] == "batch":
        refs, qs = _batch_clouds(case, gen)
        return {"refs": refs, "qs": qs}
    ref, q = _clouds(case, gen)
    out = {"ref": ref, "q": q}
    if case["op"] == "grad":
        out["w"] = _uniform(gen, case["nq"], case["k"], ref.dtype)
    elif case["op"] == "chamfer":
        out["w1"] = _uniform(gen, case["n"], case["k"], ref.dtype)
        out["w2"] = _uniform(gen, case["nq"], case["k"], ref.dtype)
    return out


def prepare(case, seed):
    state = {"case": case, **_inputs(case, seed)}
    op = case["op"]
    if op in ("grad", "chamfer"):
        state["ref"].requires_grad_(True)
        state["q"].requires_grad_(True)
    if op in ("query", "grad"):
        state["tree"] = build_kd_tree(state["ref"], levels=case.get("levels"))
    elif op == "batch":
        _, counts, ks = _batch_plan(case)
        state["tree"] = BatchedKDTrees(state["refs"], ks, counts)
        state["q"] = torch.cat(state.pop("qs"))
    return state


# ------------------------------------------------------------------ pass --

def run(state):
    case = state["case"]
    op, k = case["op"], case.get("k")
    if op == "query":
        return state["tree"].query(state["q"], nr_nns_searches=k)
    if op == "rebuild":
        return build_kd_tree(state["ref"]).query(state["q"], nr_nns_searches=k)
    if op == "grad":
        dists, inds = state["tree"].query(state["q"], nr_nns_searches=k)
        loss = 0.5 * (dists * state["w"]).sum()
        gq, gref = torch.autograd.grad(loss, (state["q"], state["ref"]))
        return dists.detach(), inds, gq, gref
    if op == "batch":
        state["tree"].query_flat(state["q"])
        return state["tree"].out_dists, state["tree"].out_idx
    if op == "chamfer":
        d1, i1, d2, i2 = nn_distance_bidirectional(state["ref"], state["q"], k)
        loss = (d1 * state["w1"]).sum() + (d2 * state["w2"]).sum()
        g1, g2 = torch.autograd.grad(loss, (state["ref"], state["q"]))
        return d1.detach(), i1, d2.detach(), i2, g1, g2
    return nn_distance(state["ref"], state["q"], k, mode=case["mode"])


# ------------------------------------------------------------------ work --

def work(case):
    """Bytes: each input read once, each output written once (a kept tree's
    points count as an input).  Flops: the distances of the neighbours that
    are returned (3 d each), which no search can do without; the exhaustive
    search of wide points, where no index saves a comparison, counts 2 d for
    every pair; a gradient counts 4 d per neighbour and cloud."""
    op = case["op"]
    s = 8 if case["dtype"] == "float64" else 4
    d = case["d"]
    if op == "batch":
        sizes, counts, ks = _batch_plan(case)
        out = sum(nq * k for nq, k in zip(counts, ks))
        return {"bytes": s * d * (sum(sizes) + sum(counts)) + (s + 4) * out, "flops": 3 * d * out}
    n, nq, k = case["n"], case["nq"], case["k"]
    pairs = nq * k
    if op == "chamfer":
        pairs = (n + nq) * k
    bytes_ = s * d * (n + nq) + (s + 4) * pairs
    flops = 3 * d * pairs
    if op == "brute" and d > 3:
        flops = 2 * d * n * nq
    if op in ("grad", "chamfer"):
        bytes_ += s * pairs + s * d * (n + nq)  # the incoming gradient, and both clouds' gradients
        flops += 8 * d * pairs
    return {"bytes": bytes_, "flops": flops}


# ----------------------------------------------------------------- exact --

PAIRS = 1 << 36  # (query, reference) pairs that plain torch compares in a few seconds


def _knn64(ref, q, k):
    """(squared distances, indices) of the k nearest in float64, sorted."""
    ref, q = ref.detach().double(), q.detach().double()
    step = max(1, (1 << 28) // ref.shape[0])
    dists, inds = [], []
    for i in range(0, q.shape[0], step):
        acc = None
        for c in range(ref.shape[1]):
            diff = q[i:i + step, c, None] - ref[None, :, c]
            acc = diff.mul_(diff) if acc is None else acc.addcmul_(diff, diff)
        dd, ii = torch.topk(acc, k, dim=1, largest=False, sorted=True)
        dists.append(dd)
        inds.append(ii)
    return torch.cat(dists), torch.cat(inds)


def _grads64(ref, q, inds, w):
    """Gradients of sum(w * squared distance) with respect to (q, ref)."""
    ref, q = ref.detach().double(), q.detach().double()
    diff = q[:, None] - ref[inds]
    g = 2.0 * w.double()[..., None] * diff
    gref = torch.zeros_like(ref).index_put_((inds.reshape(-1),), -g.reshape(-1, ref.shape[1]), accumulate=True)
    return g.sum(1), gref


def exact(case, seed):
    if case["op"] == "batch":
        sizes, counts, ks = _batch_plan(case)
        if sum(n * nq for n, nq in zip(sizes, counts)) > PAIRS:
            return None
        x = _inputs(case, seed)
        return torch.cat([_knn64(r, q, k)[0].reshape(-1) for r, q, k in zip(x["refs"], x["qs"], ks)]), None
    if case["n"] * case["nq"] > PAIRS:
        return None
    x = _inputs(case, seed)
    ref, q, k = x["ref"], x["q"], case["k"]
    if case["op"] == "chamfer":
        d1, i1 = _knn64(q, ref, k)
        d2, i2 = _knn64(ref, q, k)
        g1, g2 = _grads64(q, ref, i1, x["w1"])
        h2, h1 = _grads64(ref, q, i2, x["w2"])
        return d1, None, d2, None, g1 + h1, g2 + h2
    dists, inds = _knn64(ref, q, k)
    if case["op"] == "grad":
        gq, gref = _grads64(ref, q, inds, 0.5 * x["w"])
        return dists, None, gq, gref
    return dists, None
