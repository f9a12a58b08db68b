"""The small-window kernel against the CPU oracle, bit for bit: sizes at the edges of its lanes, blocks and bins,
dims at the edges of its staging chunks, equal distances, and the status words of invalid input."""

import json

import numpy as np
import pytest

from tests.test_gpu_parity import _compare
from tests.test_gpu_sparse import _duplicates, _lattice, _mixture, _uniform

pytestmark = pytest.mark.gpu

SIZES = [2, 3, 4, 5, 7, 8, 9, 15, 16, 17, 31, 32, 33, 47, 48, 49, 50, 63, 64, 65, 95, 96, 97, 127, 128, 129]


@pytest.mark.parametrize("precision", ["float32", "float64"])
@pytest.mark.parametrize("dims", [1, 4, 15, 16, 17, 31, 32, 33, 64, 100])
def test_sizes_and_dims(cuda, precision, dims):
    rng = np.random.default_rng(dims)
    for maker in (_mixture, _lattice):
        _compare([maker(rng, n, dims) for n in SIZES], 3, 2, 0.1, precision)


@pytest.mark.parametrize("precision", ["float32", "float64"])
@pytest.mark.parametrize("ms", [1, 3, 5, 16, 17, 31, 32, 64, 128])
def test_core_distances(cuda, precision, ms):
    rng = np.random.default_rng(ms)
    for maker in (_uniform, _duplicates):
        _compare([maker(rng, n, 3) for n in SIZES if n >= ms] or [maker(rng, ms, 3)], 2, ms, 0.0, precision)


@pytest.mark.parametrize("precision", ["float32", "float64"])
def test_invalid_values(cuda, precision):
    import torch

    from hdbscan_gb300 import hdbscan
    from hdbscan_gb300._cuda import Plan

    dtype = torch.float32 if precision == "float32" else torch.float64
    X = torch.randn(3, 24, 5, dtype=dtype, device="cuda")
    plan = Plan(np.arange(4) * 24, 5, precision=precision)
    assert {c["variant"] for c in json.loads(plan.describe())["classes"]} == {"small"}
    bad = X.clone()
    bad[1, 3, 2] = float("nan")
    with pytest.raises(ValueError, match="finite"):
        hdbscan(bad, precision=precision)
    bad = X.clone()
    bad[2, 0, 0] = torch.finfo(dtype).max
    bad[2, 1, 0] = -torch.finfo(dtype).max
    with pytest.raises(ValueError, match="overflow"):
        hdbscan(bad, precision=precision)
