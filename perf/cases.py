"""What a program clusters with this package, as timed cases.

Every case is one call through the public entry points (`hdbscan`,
`hdbscan_ragged`, `merge_weights` and autograd) on device-resident input.  The
windows are seeded mixtures of Gaussian clusters with uniform background
noise: the distributions of the benchmark workloads in
`hdbscan_gb300/synthetic.py`, drawn on the GPU so that many batches can be
made quickly.  `listed()` names the cases; `draw()` spreads over the same
ranges: 16 to 4096 points a window, 1 to 512 windows, 2 to 768 dimensions, both
precisions, half-precision embeddings, forward and backward.
"""

import math

import numpy as np
import torch

from hdbscan_gb300 import hdbscan, hdbscan_ragged, merge_weights

_DTYPES = {"float32": torch.float32, "float64": torch.float64, "bfloat16": torch.bfloat16,
           "float16": torch.float16}


def _case(name, kind, windows, low, high, dims, **options):
    """kind: 'dense' (hdbscan on [B, N, D] or [N, D]), 'ragged' (hdbscan_ragged), 'tree' (hdbscan_ragged with
    the hierarchy) or 'grad' (merge_weights and its gradient).  Window sizes: `low` when low == high, else
    log-uniform (spread 'log') or uniform in [low, high]."""
    case = {"name": name, "kind": kind, "windows": windows, "low": low, "high": high, "dims": dims,
            "precision": "float32", "input": "", "mcs": 5, "ms": 5, "eps": 0.0, "method": "eom",
            "probabilities": False, "normalize": False, "spread": "log", "sizes_seed": 1, "data": "mixture"}
    case.update(options)
    case["input"] = case["input"] or case["precision"]
    return case


def listed():
    return [
        # One small set of points clustered on its own with the default parameters: an interactive call,
        # where launches and the serial chain are all that counts.
        _case("one_100x4_f32", "dense", 1, 100, 100, 4),
        # The first benchmark workload: one float64 window, as scikit-learn's users call it.
        _case("one_512x8_f64", "dense", 1, 512, 512, 8, precision="float64"),
        # One large window, odd in size, of embedding-like points: the longest serial chain a call can have.
        _case("one_4001x32_f32", "dense", 1, 4001, 4001, 32, mcs=10, ms=10, eps=0.05, data="sphere"),
        # The batch that the reference publishes its numbers on: 32 windows of 1024 x 8 in float64, mcs = ms = 2.
        _case("batch_32x1024x8_f64", "dense", 32, 1024, 1024, 8, precision="float64", mcs=2, ms=2, eps=0.1),
        # The uniform benchmark batch: 256 windows of 1024 x 16 float32.
        _case("batch_256x1024x16_f32", "dense", 256, 1024, 1024, 16, mcs=2, ms=2, eps=0.1),
        # Encoder embeddings in bfloat16, normalised, with membership strengths: wide points, odd size.
        _case("embed_48x999x384_bf16", "dense", 48, 999, 999, 384, input="bfloat16", normalize=True, mcs=10, ms=10,
              probabilities=True, data="sphere"),
        # Heavily smoothed densities (large min_samples), leaf clusters.
        _case("smooth_24x1500x16_f32", "dense", 24, 1500, 1500, 16, mcs=25, ms=100, method="leaf"),
        # Very many tiny sets (per-user or per-document groups), float64, with the hierarchy read back.
        _case("tree_1500x16to200x6_f64", "tree", 1500, 16, 200, 6, precision="float64", mcs=4, ms=4),
        # The ragged benchmark workload: 512 windows of 64 to 4096 points, float32.
        _case("ragged_512_f32", "ragged", 512, 64, 4096, 32, mcs=10, ms=10, eps=0.05, data="sphere"),
        # The same in float64, a quarter of the windows.
        _case("ragged_128_f64", "ragged", 128, 64, 4096, 32, precision="float64", mcs=10, ms=10, eps=0.05,
              data="sphere", sizes_seed=2),
        # Training through the merge weights: forward and backward, the differentiation workload.
        _case("grad_64x2048x64_f32", "grad", 64, 2048, 2048, 64, mcs=15, ms=5),
        # The large ragged float64 workload, forward and backward: the largest call.
        _case("grad_96x2048to4096x128_f64", "grad", 96, 2048, 4096, 128, precision="float64", mcs=32, ms=16,
              spread="uniform", data="anisotropic"),
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["dense", "dense", "dense", "ragged", "ragged", "tree", "grad"])
    precision = rng.choice(["float32", "float32", "float64"])
    dims = _log_int(rng, 2, 768 if kind == "dense" else 160)
    high = _log_int(rng, 16, 4096)
    low = high if kind in ("dense", "grad") else _log_int(rng, 16, high)
    # No more coordinate pairs than the largest listed case has (96 windows of about 3072 points at 128 dims).
    budget = (4e9 if precision == "float64" else 2e10) / (high * high * dims)
    windows = max(1, min(512, _log_int(rng, 1, 512), int(budget)))
    ms = min(low, rng.choice([1, 2, 2, 3, 5, 5, 10, 16, _log_int(rng, 2, 128)]))
    case = _case("", kind, windows, low, high, dims, precision=precision, ms=ms, mcs=max(2, rng.choice([2, 5, ms, 30])),
                 eps=rng.choice([0.0, 0.0, 0.05, 0.1]), sizes_seed=rng.randrange(1 << 20),
                 spread=rng.choice(["log", "uniform"]), data=rng.choice(["mixture", "sphere", "anisotropic"]))
    if kind == "dense":
        case["method"] = rng.choice(["eom", "eom", "leaf"])
        case["probabilities"] = rng.random() < 0.25
        if precision == "float32" and rng.random() < 0.3:
            case["input"] = rng.choice(["bfloat16", "float16"])
            case["normalize"] = rng.random() < 0.5
    del case["name"]
    return case


def _sizes(case):
    low, high, windows = case["low"], case["high"], case["windows"]
    if low == high:
        return np.full(windows, low, dtype=np.int64)
    rng = np.random.default_rng(case["sizes_seed"])
    if case["spread"] == "log":
        sizes = np.rint(np.exp(rng.uniform(np.log(low), np.log(high), windows)))
    else:
        sizes = rng.integers(low, high + 1, windows)
    return np.clip(sizes, low, high).astype(np.int64)


def _points(case, seed, sizes):
    """Packed points on the GPU: per window a mixture of 4 to 20 clusters plus background noise."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    host = np.random.default_rng(int(seed))
    dims, windows, total = case["dims"], len(sizes), int(sizes.sum())
    double = dict(dtype=torch.float64, device="cuda")
    window = torch.repeat_interleave(torch.arange(windows, device="cuda"), torch.as_tensor(sizes, device="cuda"))
    clusters = torch.as_tensor(host.integers(4, 21, windows), device="cuda")
    which = torch.minimum((torch.rand(total, generator=gen, **double) * clusters[window]).long(), clusters[window] - 1)
    noise = torch.rand(total, generator=gen, **double) < (0.05 if case["data"] == "sphere" else 0.08)
    normal = torch.randn(total, dims, generator=gen, **double)
    if case["data"] == "sphere":  # L2-normalised embeddings: angular std 0.15, uniform directions as noise
        centres = torch.nn.functional.normalize(torch.randn(windows, 20, dims, generator=gen, **double), dim=2)
        points = torch.where(noise[:, None], normal, centres[window, which] + 0.15 * normal)
        points = torch.nn.functional.normalize(points, dim=1)
    else:
        centres = (torch.rand(windows, 20, dims, generator=gen, **double) - 0.5) * 8.0
        if case["data"] == "anisotropic":
            std = (0.1 + 0.9 * torch.rand(windows, 20, dims, generator=gen, **double))[window, which]
        else:
            std = (0.2 + 0.6 * torch.rand(windows, 20, 1, generator=gen, **double))[window, which]
        background = (torch.rand(total, dims, generator=gen, **double) - 0.5) * 12.0
        points = torch.where(noise[:, None], background, centres[window, which] + std * normal)
    return points.to(_DTYPES[case["input"]]).contiguous()


def prepare(case, seed):
    sizes = _sizes(case)
    offsets = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    X = _points(case, seed, sizes)
    if case["kind"] == "dense":
        X = X.view(-1, case["dims"]) if case["windows"] == 1 else X.view(case["windows"], case["low"], case["dims"])
    if case["kind"] == "grad":
        X = X.to(_DTYPES[case["precision"]]).requires_grad_(True)
    return {"case": case, "X": X, "offsets": offsets}


def run(state):
    case, X, offsets = state["case"], state["X"], state["offsets"]
    options = dict(min_cluster_size=case["mcs"], min_samples=case["ms"], cluster_selection_epsilon=case["eps"],
                   precision=case["precision"])
    if case["kind"] == "grad":
        # Total persistence of degree 2 as the loss.
        weights, labels = merge_weights(X, offsets, **options)
        (gradient,) = torch.autograd.grad(weights.square().sum(), X)
        return {"labels": labels, "weights": weights.detach(), "gradient": gradient}
    if case["kind"] == "dense":
        result = hdbscan(X, cluster_selection_method=case["method"], return_probabilities=case["probabilities"],
                         normalize=case["normalize"], **options)
        return {"labels": result[0], "probabilities": result[1]} if case["probabilities"] else {"labels": result}
    if case["kind"] == "ragged":
        return {"labels": hdbscan_ragged(packed=X, offsets=offsets, **options)[0]}
    labels, _, tree = hdbscan_ragged(packed=X, offsets=offsets, return_hierarchy=True, **options)
    out = {"labels": labels}
    for name in ("edges_uv", "edge_w", "order", "link_lr", "link_w", "link_size", "n_clusters", "point_parent",
                 "point_lambda", "core", "probabilities"):
        if name in tree:
            out[name] = tree[name]
    return out


def work(case):
    sizes = _sizes(case).astype(float)
    total, pairs = sizes.sum(), (sizes * (sizes - 1) / 2).sum()
    element = {"float64": 8, "float32": 4}.get(case["input"], 2)
    real = 8 if case["precision"] == "float64" else 4
    moved = total * case["dims"] * element + 4 * total  # points in, labels out
    flops = 3.0 * case["dims"] * pairs  # one difference, square and sum a pair and coordinate
    if case["probabilities"]:
        moved += real * total
    if case["kind"] == "tree":
        moved += total * (8 + real + 4 + 8 + real + 4 + 4 + real + real) + (real * total if case["ms"] > 2 else 0)
    if case["kind"] == "grad":
        moved += real * total * (2 + 2 * case["dims"])  # weights and their gradient, points again, gradient out
        flops += 5.0 * case["dims"] * total
    return {"bytes": float(moved), "flops": float(flops)}


def _exact_windows(x, sizes, ms):
    """Per window (sorted merge weights, pair of points behind each, core distances or None) in float64, for a
    list of windows at once: x [B, n, D], padded; sizes [B]."""
    B, n, _ = x.shape
    dev = x.device
    sizes = torch.as_tensor(sizes, device=dev)
    rows = torch.arange(B, device=dev)
    inside = torch.arange(n, device=dev)[None] < sizes[:, None]
    d = torch.cdist(x, x, compute_mode="donot_use_mm_for_euclid_dist")
    d.masked_fill_(~inside[:, None, :], float("inf"))
    core = nbr = None
    if ms > 2:
        value, index = torch.topk(d, ms, dim=2, largest=False, sorted=True)
        core, nbr = value[..., -1].contiguous(), index[..., -1].contiguous()
    best = torch.full((B, n), float("inf"), dtype=d.dtype, device=dev)
    source = torch.zeros((B, n), dtype=torch.long, device=dev)
    outside = inside.clone()
    order, sources = (torch.zeros((n, B), dtype=torch.long, device=dev) for _ in range(2))
    weights = torch.full((n, B), float("inf"), dtype=d.dtype, device=dev)
    current = torch.zeros(B, dtype=torch.long, device=dev)
    for i in range(n):  # Prim, one step of every window at a time
        outside[rows, current] = False
        order[i], weights[i], sources[i] = current, best[rows, current], source[rows, current]
        row = d[rows, current]
        if ms > 2:
            row = torch.maximum(row, torch.maximum(core, core[rows, current][:, None]))
        closer = row < best
        best = torch.where(closer, row, best)
        source = torch.where(closer, current[:, None], source)
        current = torch.argmin(torch.where(outside, best, float("inf")), dim=1)
    found = []
    for b, count in enumerate(sizes.tolist()):
        w, u, v = weights[1:count, b], sources[1:count, b], order[1:count, b]
        p, q = u, v
        if ms > 2:  # the distance that attains the maximum: the pair's own, else a core distance
            own, by_u = d[b][u, v] == w, core[b][u] == w
            p = torch.where(own | by_u, u, v)
            q = torch.where(own, v, torch.where(by_u, nbr[b][u], nbr[b][v]))
        w, rank = torch.sort(w, stable=True)
        found.append((w, p[rank], q[rank], None if core is None else core[b, :count]))
    return found


def exact(case, seed):
    if case["kind"] not in ("grad", "tree"):
        return None  # labels are whole numbers
    sizes = _sizes(case)
    state = prepare(case, seed)
    x, offsets = state["X"].detach().double(), state["offsets"]
    step = max(1, int(1.5e9 // int(sizes.max()) ** 2))
    if -(-len(sizes) // step) * int(sizes.max()) > 30000:
        return None  # over 20 seconds of single Prim steps
    weights, cores = [], []
    gradient = torch.zeros_like(x)
    for first in range(0, len(sizes), step):
        chunk = range(first, min(first + step, len(sizes)))
        parts = [x[offsets[w] : offsets[w + 1]] for w in chunk]
        padded = torch.nn.utils.rnn.pad_sequence(parts, batch_first=True)
        for w, part, (value, a, b, core) in zip(chunk, parts, _exact_windows(padded, sizes[chunk], case["ms"])):
            weights.append(value)
            cores.append(core)
            if case["kind"] == "grad":
                difference = part[a] - part[b]
                norm = difference.square().sum(1, keepdim=True).sqrt()
                term = torch.where(norm > 0, 2.0 * value[:, None] * difference / norm, 0.0)
                target = gradient[offsets[w] : offsets[w + 1]]
                target.index_add_(0, a, term)
                target.index_add_(0, b, -term)
    if case["kind"] == "grad":
        return {"labels": None, "weights": torch.cat(weights), "gradient": gradient}
    out = {"labels": None, "edges_uv": None, "edge_w": None, "order": None, "link_lr": None,
           "link_w": torch.cat(weights), "link_size": None, "n_clusters": None, "point_parent": None,
           "point_lambda": None, "probabilities": None}
    if case["ms"] > 2:
        out["core"] = torch.cat(cores)
    return out
