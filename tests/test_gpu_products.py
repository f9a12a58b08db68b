"""The sparse path on tensor-core products against the CPU oracle, bit for bit, for both precisions over the dims and
list lengths that take products; data that the bound cannot separate included.  Invalid values end in the general
path's status words."""

import json

import numpy as np
import pytest

from oracle import oracle
from tests.test_gpu_sparse import MAKERS, _mixture, zlib_seed

pytestmark = pytest.mark.gpu

STAGES = (("edges_uv", 1), ("edge_w", 1), ("order", 1), ("link_lr", 1), ("link_w", 1), ("link_size", 1), ("labels", 0),
          ("point_parent", 0))


def _plan(offsets, dims, precision, mcs=5, ms=5, eps=0.0):
    from hdbscan_gb300 import _lib
    from hdbscan_gb300._cuda import Plan

    plan = Plan(offsets, dims, min_cluster_size=mcs, min_samples=ms, cluster_selection_epsilon=eps, precision=precision,
                test_flags=_lib.HDB_FLAG_FORCE_PRODUCTS)
    describe = json.loads(plan.describe())
    assert describe["products"]
    return plan, describe


def _check(windows, mcs, ms, eps, precision):
    import torch

    from hdbscan_gb300._cuda import pack

    dtype = np.float32 if precision == "float32" else np.float64
    windows = [np.asarray(x, dtype) for x in windows]
    packed, offsets = pack(windows, precision)
    plan, describe = _plan(offsets, packed.shape[1], precision, mcs, ms, eps)
    workspace = plan.workspace()
    buffers = plan.export_buffers(hierarchy=True, gradients=True, probabilities=True)
    labels, status = plan.forward(packed, workspace=workspace, exports=buffers)
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    host = {k: v.cpu().numpy() for k, v in buffers.items()}
    host["labels"] = labels.cpu().numpy()
    for w, x in enumerate(windows):
        o = oracle.cluster(x, mcs, ms, eps, precision)
        lo, hi = offsets[w], offsets[w + 1]
        for name, edges in STAGES + ((("core", 0),) if ms > 2 else ()):
            part = slice(lo - w, hi - w - 1) if edges else slice(lo, hi)
            got, want = np.ascontiguousarray(host[name][part]), np.ascontiguousarray(o[name])
            np.testing.assert_array_equal(got.view(np.uint8), want.astype(got.dtype).view(np.uint8),
                                          err_msg=f"window {w} n={len(x)} d={x.shape[1]} ms={ms} {precision}: {name}")
    return describe


@pytest.mark.parametrize("ms", [2, 5, 17])
@pytest.mark.parametrize("dims", [32, 33, 65, 384])
@pytest.mark.parametrize("maker", sorted(MAKERS))
@pytest.mark.parametrize("precision", ["float32", "float64"])
def test_data_and_dims(cuda, maker, dims, ms, precision):
    if precision == "float32" and maker == "huge":
        pytest.skip("squares overflow float32")
    rng = np.random.default_rng(zlib_seed(maker, dims + ms))
    sizes = (384, 385, 517) if precision == "float32" else (33, 64, 129, 517)
    _check([MAKERS[maker](rng, n, dims) for n in sizes], 4, ms, 0.05, precision)


@pytest.mark.parametrize("maker", ["mixture", "far", "duplicates", "tiny"])
@pytest.mark.parametrize("dims", [768, 1024, 2048])
@pytest.mark.parametrize("precision", ["float32", "float64"])
def test_many_dims(cuda, maker, dims, precision):
    rng = np.random.default_rng(dims)
    _check([MAKERS[maker](rng, 400, dims)], 4, 5, 0.0, precision)


# Lists of 8, 16, 32 and 64 entries and their ends (the last ms with a list of each length, and the next).
@pytest.mark.parametrize("ms", [1, 3, 4, 5, 6, 17, 18, 40, 57, 58, 59])
@pytest.mark.parametrize("maker", ["mixture", "uniform", "duplicates"])
@pytest.mark.parametrize("precision", ["float32", "float64"])
def test_list_lengths(cuda, maker, ms, precision):
    rng = np.random.default_rng(ms)
    if ms == 59:  # no list: the general path
        from hdbscan_gb300 import _lib
        from hdbscan_gb300._cuda import Plan

        plan = Plan(np.arange(2) * 900, 40, min_samples=ms, precision=precision, test_flags=_lib.HDB_FLAG_FORCE_PRODUCTS)
        assert not json.loads(plan.describe())["products"]
        return
    _check([MAKERS[maker](rng, n, 40) for n in (400, 900)], 6, ms, 0.0, precision)


def test_window_near_the_largest(cuda):
    rng = np.random.default_rng(3)
    _check([_mixture(rng, n, 48) for n in (4096, 4095)], 10, 10, 0.0, "float32")


@pytest.mark.parametrize("products", [True, False])
@pytest.mark.parametrize("value", ["nan", "inf", "overflow"])
@pytest.mark.parametrize("precision", ["float32", "float64"])
def test_invalid_values(cuda, precision, value, products):
    # The middle window is invalid; the others keep their labels.
    import torch

    from hdbscan_gb300 import _lib
    from hdbscan_gb300._cuda import Plan

    dtype = torch.float32 if precision == "float32" else torch.float64
    dims = 40 if products or precision == "float32" else 20
    n = 600
    rng = np.random.default_rng(1)
    X = torch.as_tensor(np.concatenate([_mixture(rng, n, dims) for _ in range(3)])).to(dtype).cuda()
    top = torch.finfo(dtype).max
    if value == "overflow":
        X[n + 5, 3], X[n + 500, 3] = top, -top
    else:
        X[n + 5, 3] = float(value)
    got = []
    for flags in (_lib.HDB_FLAG_FORCE_PRODUCTS if products else 0, _lib.HDB_FLAG_NO_SPARSE):
        for ms in (2, 5):
            plan = Plan(np.arange(4) * n, dims, min_samples=ms, precision=precision, test_flags=flags)
            describe = json.loads(plan.describe())
            assert any(c["variant"] == "sparse" for c in describe["classes"]) == (flags != _lib.HDB_FLAG_NO_SPARSE)
            labels, status = plan.forward(X)
            got.append((int(status.item()), labels.cpu().numpy()))
    for (status, labels), (want_status, want_labels) in zip(got[:2], got[2:]):
        for word in (status, want_status):  # a value that is not finite may set the overflow bit as well
            if value == "overflow":
                assert word == _lib.STATUS_OVERFLOW
            else:
                assert word & _lib.STATUS_NONFINITE
        np.testing.assert_array_equal(labels, want_labels)
        assert (labels[n:2 * n] == -1).all() and (labels[:n] >= 0).any()
