"""Core distances beyond the neighbour lists (select kernel, several rows a CTA) against the CPU oracle, bit for bit.

Sizes leave ragged row groups (8, 4, 2 and 1 rows a CTA by window size); lattices give many equal distances, whose
neighbour is the one of lowest index; widely scaled points spread the keys over their whole range.
"""

import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


def _lattice(rng, n, d):
    return rng.integers(-2, 3, (n, d)) / 2.0


def _scaled(rng, n, d):
    return rng.normal(size=(n, d)) * np.exp(rng.uniform(-12, 12, (n, 1)))


@pytest.mark.parametrize("precision", ["float32", "float64"])
@pytest.mark.parametrize("dims", [3, 40])
@pytest.mark.parametrize("maker", [_lattice, _scaled])
@pytest.mark.parametrize("sizes,ms", [((65, 66, 71, 200), 65), ((1025, 2051), 100), ((4095, 4096), 127)])
def test_core_distances_and_neighbours(cuda, precision, dims, maker, sizes, ms):
    import torch

    from hdbscan_gb300._cuda import Plan, pack

    dtype = np.float32 if precision == "float32" else np.float64
    rng = np.random.default_rng(sizes[0] + ms + dims)
    windows = [maker(rng, n, dims).astype(dtype) for n in sizes]
    packed, offsets = pack(windows, precision)
    plan = Plan(offsets, dims, min_cluster_size=5, min_samples=ms, precision=precision)
    buffers = plan.export_buffers(hierarchy=True, gradients=True)
    labels, status = plan.forward(packed, exports=buffers)
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    core, nbr = buffers["core"].cpu().numpy(), buffers["core_nbr"].cpu().numpy()
    for w, x in enumerate(windows):
        part = slice(offsets[w], offsets[w + 1])
        want = oracle.cluster(x, 5, ms, 0.0, precision)
        np.testing.assert_array_equal(core[part].view(np.uint8), want["core"].view(np.uint8))
        np.testing.assert_array_equal(labels[offsets[w]:offsets[w + 1]].cpu().numpy(), want["labels"])
        # The neighbour's own distance is the core distance, and fewer than ms points come before it.
        for i in range(0, len(x), max(1, len(x) // 50)):
            d = np.zeros(len(x), dtype)
            for k in range(dims):
                delta = (x[i, k] - x[:, k]).astype(dtype)
                d = (d + (delta * delta).astype(dtype)).astype(dtype)
            d = np.sqrt(d).astype(dtype)
            order = np.lexsort((np.arange(len(x)), d))
            assert nbr[part][i] == order[ms - 1], (w, i)
