"""Windows built against the error bound of the sparse path's distances, bit for bit against the CPU oracle.

Each set makes one share of the error as large as it gets; a bound without that share gives a wrong core distance
and no fallback.
"""

import json

import numpy as np
import pytest

from tests.test_gpu_sparse import _check

pytestmark = pytest.mark.gpu


def rounding_window(n=2048, d=1024):
    """float32 sums of squares that round far apart: one point's neighbours lie at a squared distance of 4 and a
    little.  Eight of them add that little in one coordinate (kept), one adds half a unit of 4's last place in every
    coordinate (each rounded away): the farthest of the nine, by (d - 1) / 2 units, is the nearest in float32."""
    rng = np.random.default_rng(7)
    x = np.zeros((n, d))
    # The rest: groups of about 16, each away from all others, with nothing undecided inside.
    unit = rng.normal(0, 1 / np.sqrt(d), (n + n // 16, d - 1))
    x[:, 1:] = 2 * unit[n + rng.integers(0, n // 16, n)] + rng.uniform(0.1, 1, (n, 1)) * unit[:n]
    x[:, 0] = 1.0
    samples = np.arange(16) * n // 16  # where the path takes its centre: their mean is zero
    far = rng.normal(0, 1, (8, d - 1))
    far *= 3 / np.linalg.norm(far, axis=1, keepdims=True)
    x[samples[:8], 1:], x[samples[8:], 1:] = far, -far
    x[samples, 0] = np.where(np.arange(16) % 2 == 0, 1.0, -1.0)
    free = np.setdiff1d(np.arange(n), samples)
    place = rng.choice(free, 10, replace=False)
    x[place] = 0.0
    x[place[0], 0] = -1.0  # the point whose neighbours these are
    x[place[1:], 0] = 1.0
    x[place[1:9], 1] = np.sqrt(2.0 ** -21 * 2 * np.arange(1, 9))
    x[place[9], 1:] = 2.0 ** -11
    return x.astype(np.float32)


def tiny_window(n=3000, d=32):
    """A float64 cluster so small that the squares of its points' coordinates have no place in float32, in a window of ordinary
    range whose centre lies in that cluster."""
    rng = np.random.default_rng(11)
    x = rng.uniform(-4, 4, (8, d))[rng.integers(0, 8, n)] + rng.normal(0, 0.5, (n, d))
    samples = np.arange(16) * n // 16
    others = rng.choice(np.setdiff1d(np.arange(n), samples), 24, replace=False)
    x[np.concatenate([samples, others])] = rng.normal(0, 1, (40, d)) * 2e-22 / np.sqrt(d)
    return x


def test_rounding_of_the_exact_sum(cuda):
    _check([rounding_window()], 5, 5, 0.0, "float32")


def test_squares_below_float32(cuda):
    _check([tiny_window()], 5, 5, 0.0, "float64")


@pytest.mark.parametrize("d, sparse", [(1 << 16, True), ((1 << 16) + 1, False)])
def test_most_dims_of_narrowed_points(cuda, d, sparse):
    rng = np.random.default_rng(d)
    describe, _ = _check([rng.normal(size=(40, d))], 4, 3, 0.0, "float64")
    assert any(c["variant"] == "sparse" for c in describe["classes"]) == sparse


def one_coordinate(windows, n, d, seed):
    """Points on an axis: what bfloat16 pairs leave of them is one coordinate's rounding, which nothing averages."""
    rng = np.random.default_rng(seed)
    x = np.zeros((windows, n, d))
    x[:, :, 0] = np.cumsum(1.0 + 0.3 * rng.random((windows, n)), axis=1)
    return rng.permuted(x, axis=1)


@pytest.mark.parametrize("precision, d, ms", [("float64", 32, 28)] + [
    (p, d, ms) for p in ("float32", "float64") for d, ms in ((37, 28), (64, 10), (64, 22))])
def test_rounding_of_bfloat16_pairs(cuda, precision, d, ms):
    import torch

    from hdbscan_gb300 import _lib
    from hdbscan_gb300._cuda import Plan

    windows, n = 300, 900
    X = torch.as_tensor(one_coordinate(windows, n, d, d + ms).reshape(-1, d)).to(getattr(torch, precision)).cuda()
    outputs = []
    for flags in (_lib.HDB_FLAG_FORCE_PRODUCTS, _lib.HDB_FLAG_NO_SPARSE):
        plan = Plan(np.arange(windows + 1) * n, d, min_cluster_size=5, min_samples=ms, precision=precision, test_flags=flags)
        assert json.loads(plan.describe())["products"] == (flags == _lib.HDB_FLAG_FORCE_PRODUCTS)
        buffers = plan.export_buffers(hierarchy=False, gradients=True)
        labels, status = plan.forward(X, exports=buffers)
        assert int(status.item()) == 0
        outputs.append(dict(buffers, labels=labels))
    for name in outputs[0]:
        got, want = (o[name].contiguous().view(torch.uint8) for o in outputs)
        assert torch.equal(got, want), name
