"""Windows that leave the sparse path: the same outputs as without it, in about the same time, in the variants that
they have without it."""

import json

import numpy as np
import pytest

from tests.test_gpu_sparse import _mixture

pytestmark = pytest.mark.gpu


def _plan(sizes, dims, ms, precision, flags=0, mcs=5):
    from hdbscan_gb300._cuda import Plan

    offsets = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    return Plan(offsets, dims, min_cluster_size=mcs, min_samples=ms, precision=precision, test_flags=flags)


def _forward(plan, X):
    """All outputs of a forward, and the flags of its windows."""
    import torch

    workspace = plan.workspace()
    buffers = plan.export_buffers(hierarchy=True, gradients=True, probabilities=True)
    for value in buffers.values():
        value.zero_()
    labels, status = plan.forward(X, workspace=workspace, exports=buffers)
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    at = json.loads(plan.describe())["general_flags_offset"]
    flags = None if at < 0 else workspace[at:at + 4 * plan.windows].view(torch.int32).cpu().numpy()
    return dict(buffers, labels=labels), flags


def _assert_same(a, b):
    import torch

    for name in a:
        assert torch.equal(a[name].contiguous().view(torch.uint8), b[name].contiguous().view(torch.uint8)), name


def _milliseconds(plan, X):
    import torch

    workspace = plan.workspace()
    times = []
    for _ in range(7):
        start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        start.record()
        plan.forward(X, workspace=workspace)
        end.record()
        end.synchronize()
        times.append(start.elapsed_time(end))
    return float(np.median(times[2:]))


def _repeated(rng, n, dims, copies):
    x = _mixture(rng, -(-n // copies), dims)
    return np.tile(x, (copies, 1))[rng.permutation(len(x) * copies)[:n]]


def _tied(dims, copies, n_max=None):
    """`copies` of every unit vector: all distances but zero are equal."""
    return np.repeat(np.eye(dims), copies, axis=0)[:n_max]


@pytest.mark.parametrize("count", [1, 2, 7, 300])
@pytest.mark.parametrize("precision", ["float32", "float64"])
def test_windows_that_leave_early_and_late(cuda, precision, count):
    # 10 copies of a point outnumber the neighbour lists (flag 1); of equal distances between groups of 6 there are
    # more than the light edges held (flag 2).  300: more windows than one pass over the flags takes.
    import torch

    from hdbscan_gb300 import _lib

    rng = np.random.default_rng(count)
    dims = 80 if count < 300 else 66
    kinds = [(2, _tied(dims, 6)), (1, _tied(dims, 10, 6 * dims)), (0, _mixture(rng, 6 * dims, dims))]
    order = [(w * w + w // 3) % 3 for w in range(count)]
    windows = [kinds[i][1][rng.permutation(6 * dims)] for i in order]
    X = torch.as_tensor(np.concatenate(windows)).to(getattr(torch, precision)).cuda()
    sizes = [len(x) for x in windows]
    got, flags = _forward(_plan(sizes, dims, 5, precision), X)
    want, _ = _forward(_plan(sizes, dims, 5, precision, _lib.HDB_FLAG_NO_SPARSE), X)
    np.testing.assert_array_equal(flags, [kinds[i][0] for i in order])
    _assert_same(got, want)


@pytest.mark.parametrize("ms", [4, 16])
def test_many_small_windows(cuda, ms):
    import torch

    from hdbscan_gb300 import _lib

    rng = np.random.default_rng(5)
    sizes = rng.integers(33, 201, 1100)
    X = torch.as_tensor(np.concatenate([_repeated(rng, n, 6, 2 + 10 * (w % 3 > 0) + ms)
                                        for w, n in enumerate(sizes)])).cuda()
    sparse, general = _plan(sizes, 6, ms, "float64"), _plan(sizes, 6, ms, "float64", _lib.HDB_FLAG_NO_SPARSE)
    got, flags = _forward(sparse, X)
    want, _ = _forward(general, X)
    assert (flags != 0).mean() > 0.5
    _assert_same(got, want)
    # (All on the CTAs that one window's tiles and rows keep busy: 20 times as long.)
    assert _milliseconds(sparse, X) < 3 * _milliseconds(general, X)


@pytest.mark.parametrize("precision, sizes, dims", [
    ("float32", [999] * 48, 384), ("float32", [2048] * 32, 64), ("float64", [1024] * 32, 8), ("float64", [2048] * 24, 64),
    ("float64", [4000, 2500, 1300, 700, 300], 32)])
def test_repeated_rows(cuda, precision, sizes, dims):
    import torch

    from hdbscan_gb300 import _lib

    rng = np.random.default_rng(dims)
    X = torch.as_tensor(np.concatenate([_repeated(rng, n, dims, 20) for n in sizes])).to(getattr(torch, precision)).cuda()
    sparse, general = _plan(sizes, dims, 5, precision), _plan(sizes, dims, 5, precision, _lib.HDB_FLAG_NO_SPARSE)
    got, flags = _forward(sparse, X)
    want, _ = _forward(general, X)
    assert flags.all()
    _assert_same(got, want)
    assert _milliseconds(sparse, X) < 1.6 * _milliseconds(general, X)


@pytest.mark.parametrize("precision", ["float32", "float64"])
def test_groups_that_flag_while_others_return(cuda, precision):
    # Windows of several groups: one group's way back starts while the next one's lists are still being looked at.
    import torch

    from hdbscan_gb300 import _lib

    rng = np.random.default_rng(3)
    sizes = [int(n) for n in rng.integers(400, 3000, 40)] + [int(n) for n in rng.integers(40, 400, 200)]
    dims, ms = (40, 5) if precision == "float32" else (6, 4)
    makers = [lambda n: _mixture(rng, n, dims), lambda n: _repeated(rng, n, dims, 3), lambda n: _repeated(rng, n, dims, 20)]
    X = torch.as_tensor(np.concatenate([makers[2 if w % 37 == 0 else w % 5 // 4](n)
                                        for w, n in enumerate(sizes)])).to(getattr(torch, precision)).cuda()
    plan = _plan(sizes, dims, ms, precision)
    want, _ = _forward(_plan(sizes, dims, ms, precision, _lib.HDB_FLAG_NO_SPARSE), X)
    for _ in range(20):
        got, flags = _forward(plan, X)
        assert flags.any() and not flags.all()
        _assert_same(got, want)


def test_capture_with_flagged_windows(cuda):
    import torch

    rng = np.random.default_rng(9)
    windows = [_tied(80, 6), _tied(80, 10, 480), _mixture(rng, 480, 80)]
    X = torch.as_tensor(np.concatenate(windows)).cuda()
    plan = _plan([len(x) for x in windows], 80, 5, "float64")
    labels = plan.forward(X)[0].clone()
    plan.capture(X)
    for _ in range(3):
        replayed, status = plan.replay()
    torch.cuda.synchronize()
    assert int(status.item()) == 0 and torch.equal(labels, replayed)


@pytest.mark.parametrize("precision, n, dims, ms, cluster", [
    ("float64", 4001, 16, 100, 4), ("float64", 2000, 64, 100, 2), ("float64", 4001, 16, 10, 4), ("float32", 2000, 32, 2, 2)])
def test_cluster_rules_of_the_table(cuda, precision, n, dims, ms, cluster):
    # A cluster serves one large window on the general path; the sparse path takes the window all the same.
    from hdbscan_gb300 import _lib

    classes = json.loads(_plan([n], dims, ms, precision, _lib.HDB_FLAG_NO_SPARSE).describe())["classes"]
    assert [c["cluster"] for c in classes] == [cluster]
    classes = json.loads(_plan([n], dims, ms, precision).describe())["classes"]
    assert [c["variant"] for c in classes] == ["matrix" if ms > 64 else "sparse"]


@pytest.mark.parametrize("precision, sizes, dims, ms, sparse", [
    ("float64", [1500] * 5000, 6, 5, True),              # 90 GB of distance blocks: room for some windows
    ("float64", [1500] * 20000, 6, 5, False),            # 30 GB of arrays over all points
    ("float64", [200] * 200000, 6, 5, False),
    ("float32", [4000] + [60] * 700000, 4, 5, False),
    ("float64", [1024] * 64, 8, 5, True)])
def test_workspace_of_large_batches(cuda, precision, sizes, dims, ms, sparse):
    # The sparse path adds at most 16 GB (and its rounding) to what the batch takes without it.
    from hdbscan_gb300 import _lib

    # (Register variants, which have no blocks, as float64 windows of few dims had them.)
    from tests.test_gpu_cluster import forced_variant

    with forced_variant(precision, 512, 4, 8, 1):
        plan = _plan(sizes, dims, ms, precision)
        general = _plan(sizes, dims, ms, precision, _lib.HDB_FLAG_NO_SPARSE)
    assert plan.workspace_bytes <= general.workspace_bytes + (17 << 30)
    assert any(c["variant"] == "sparse" for c in json.loads(plan.describe())["classes"]) == sparse


@pytest.mark.parametrize("n, dims, ms, count, sparse", [
    (1023, 8, 3, 1, False), (1024, 8, 3, 24, True), (1024, 8, 3, 25, False), (1535, 8, 2, 2, False),
    (1536, 8, 2, 2, True), (4000, 8, 3, 24, True)])
def test_register_windows_on_the_sparse_path(cuda, n, dims, ms, count, sparse):
    # The rule by itself: the variant is given, whatever the table says of these sizes.
    from tests.test_gpu_cluster import forced_variant

    with forced_variant("float32", 512, 8, 8, 1, small=True):
        classes = json.loads(_plan([n] * count, dims, ms, "float32").describe())["classes"]
    assert [c["variant"] for c in classes][0] == ("sparse" if sparse else "recompute")
