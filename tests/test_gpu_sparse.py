"""The sparse path (light edges + sparse Prim) against the CPU oracle, bit for bit on every exported stage.

Sizes sit at the edges of its bins, blocks and tiles; the data include what
its float32 bound cannot separate (duplicates, lattices, tiny or huge values,
small clusters far from the origin), where windows fall back to the general
path.  Nothing here has a tolerance: integers and bit patterns are equal.
"""

import json

import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


def _mixture(rng, n, d):
    centres = rng.uniform(-4, 4, (6, d))
    x = centres[rng.integers(0, 6, n)] + rng.normal(0, 0.4, (n, d))
    x[rng.random(n) < 0.08] += rng.uniform(-6, 6, d)
    return x


def _uniform(rng, n, d):
    return rng.uniform(-1, 1, (n, d))


def _line(rng, n, d):  # neighbours in a row: long merge chains
    x = np.zeros((n, d))
    x[:, 0] = np.cumsum(1.0 + 0.3 * rng.random(n))
    return x[rng.permutation(n)]


def _nested(rng, n, d):  # growing gaps: deep dendrogram, one component swallows the rest
    x = np.zeros((n, d))
    x[:, 0] = np.cumsum(1.0 + 0.01 * np.arange(n)) + 1e-3 * rng.random(n)
    return x


def _far(rng, n, d):  # small clusters far from the origin and from each other
    return 1e6 + 1e3 * rng.integers(0, 3, (n, 1)) + rng.normal(0, 1e-3, (n, d))


def _duplicates(rng, n, d):
    return np.repeat(rng.normal(size=(n // 3 + 1, d)), 3, axis=0)[:n][rng.permutation(n)]


def _lattice(rng, n, d):
    return rng.integers(-3, 4, (n, d)) / 2.0


def _tiny(rng, n, d):
    return _mixture(rng, n, d) * 1e-30


def _huge(rng, n, d):
    return _mixture(rng, n, d) * 1e15


MAKERS = {f.__name__[1:]: f for f in (_mixture, _uniform, _line, _nested, _far, _duplicates, _lattice, _tiny, _huge)}


def _run(windows, mcs, ms, eps, precision):
    import torch

    from hdbscan_gb300._cuda import Plan, pack

    packed, offsets = pack(windows, precision)
    plan = Plan(offsets, packed.shape[1], min_cluster_size=mcs, min_samples=ms, cluster_selection_epsilon=eps,
                precision=precision)
    workspace = plan.workspace()
    buffers = plan.export_buffers(hierarchy=True, gradients=True, probabilities=True)
    labels, status = plan.forward(packed, workspace=workspace, exports=buffers)
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    host = {k: v.cpu().numpy() for k, v in buffers.items()}
    host["labels"] = labels.cpu().numpy()
    describe = json.loads(plan.describe())
    at = describe["general_flags_offset"]
    flags = None
    if at >= 0:
        flags = workspace[at:at + 4 * plan.windows].cpu().numpy().view(np.int32)
    return host, offsets, describe, flags


def _check(windows, mcs, ms, eps, precision):
    dtype = np.float32 if precision == "float32" else np.float64
    windows = [np.asarray(x, dtype) for x in windows]
    host, offsets, describe, flags = _run(windows, mcs, ms, eps, precision)
    for w, x in enumerate(windows):
        o = oracle.cluster(x, mcs, ms, eps, precision)
        lo, hi = offsets[w], offsets[w + 1]
        e0, e1 = lo - w, hi - w - 1
        ctx = f"window {w} n={len(x)} d={x.shape[1]} mcs={mcs} ms={ms} {precision}"
        for name, part in (("edges_uv", slice(e0, e1)), ("edge_w", slice(e0, e1)), ("order", slice(e0, e1)),
                           ("link_lr", slice(e0, e1)), ("link_w", slice(e0, e1)), ("link_size", slice(e0, e1)),
                           ("labels", slice(lo, hi)), ("point_parent", slice(lo, hi))) + (
                               (("core", slice(lo, hi)),) if ms > 2 else ()):
            got, want = np.ascontiguousarray(host[name][part]), np.ascontiguousarray(o[name])
            np.testing.assert_array_equal(got.view(np.uint8), want.astype(got.dtype).view(np.uint8),
                                          err_msg=f"{ctx}: {name}")
    return describe, flags


@pytest.mark.parametrize("ms", [1, 2, 3, 5, 6, 7, 14, 15, 16])
@pytest.mark.parametrize("maker", sorted(MAKERS))
@pytest.mark.parametrize("precision", ["float32", "float64"])
def test_sizes_and_data(cuda, maker, ms, precision):
    rng = np.random.default_rng(zlib_seed(maker, ms))
    sizes = [15, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 257, 511, 512, 513]
    d = int(rng.integers(1, 20)) if precision == "float64" else 33  # float32: the matrix variant's dims
    if precision == "float32" and maker == "huge":
        pytest.skip("squares overflow float32")
    describe, flags = _check([MAKERS[maker](rng, max(n, ms), d) for n in sizes], 4, ms, 0.05, precision)
    assert any(c["variant"] == "sparse" for c in describe["classes"])
    if maker in ("mixture", "uniform"):
        assert not flags.any(), "ordinary data stays on the sparse path"


def zlib_seed(name, ms):
    import zlib

    return zlib.crc32(f"{name}/{ms}".encode())


@pytest.mark.parametrize("precision", ["float32", "float64"])
@pytest.mark.parametrize("dims", [1, 2, 31, 32, 33, 64, 65, 129, 300])
def test_dimensions(cuda, dims, precision):
    rng = np.random.default_rng(dims)
    _check([_mixture(rng, n, dims) for n in (100, 260, 700)], 5, 5, 0.0, precision)


@pytest.mark.parametrize("precision", ["float32", "float64"])
@pytest.mark.parametrize("ms", [2, 16])
@pytest.mark.parametrize("n", [1023, 1024, 1025, 2047, 2048, 2049, 4095, 4096])
def test_large_windows(cuda, n, ms, precision):
    rng = np.random.default_rng(n + ms)
    d = 9 if precision == "float64" else 40
    _check([_mixture(rng, n, d), _uniform(rng, n, d)], 8, ms, 0.0, precision)


@pytest.mark.parametrize("precision", ["float32", "float64"])
@pytest.mark.parametrize("ms", [30, 31, 62, 63, 64])
def test_long_lists(cuda, ms, precision):
    rng = np.random.default_rng(ms)
    d = 7 if precision == "float64" else 70
    _check([_mixture(rng, n, d) for n in (ms, ms + 1, 200, 900)], 10, ms, 0.0, precision)


@pytest.mark.parametrize("precision", ["float32", "float64"])
def test_many_flagged_windows(cuda, precision):
    # More distance tiles and rows on the general path than one pass of its fixed grids holds.
    rng = np.random.default_rng(99)
    # (Every point 50 times: no list can reach past its copies.)
    windows = [np.repeat(rng.normal(size=(22 + i % 5, 36)), 50, axis=0) for i in range(40)]
    windows += [_mixture(rng, 700, 36) for _ in range(3)]
    dtype = np.float32 if precision == "float32" else np.float64
    host, offsets, describe, flags = _run([x.astype(dtype) for x in windows], 5, 6, 0.0, precision)
    assert flags[:40].all() and not flags[40:].any()
    for w in (0, 7, 23, 39, 40, 42):
        o = oracle.cluster(windows[w].astype(dtype), 5, 6, 0.0, precision)
        lo, hi = offsets[w], offsets[w + 1]
        np.testing.assert_array_equal(host["edges_uv"][lo - w:hi - w - 1], o["edges_uv"])
        np.testing.assert_array_equal(host["core"][lo:hi].view(np.uint8), o["core"].view(np.uint8))
        np.testing.assert_array_equal(host["labels"][lo:hi], o["labels"])


@pytest.mark.parametrize("n, dims, ms, count, sparse", [
    (1023, 16, 3, 1, False), (1024, 16, 3, 1, True), (1024, 16, 3, 24, True), (1024, 16, 3, 25, False),
    (1535, 4, 2, 2, False), (1536, 4, 2, 2, True), (511, 17, 4, 2, False), (512, 17, 4, 2, True),
    (1536, 32, 3, 25, True), (2049, 2, 5, 1, True), (3000, 8, 2, 1, True)])
def test_few_windows_of_few_dims(cuda, n, dims, ms, count, sparse):
    # float32 windows whose coordinates the general form keeps in registers.
    rng = np.random.default_rng(n + dims)
    windows = [(_mixture, _lattice)[w % 2](rng, n, dims) for w in range(count)]
    describe, _ = _check(windows, 5, ms, 0.0, "float32")
    if sparse or all(c["variant"] != "matrix" for c in describe["classes"]):
        assert any(c["variant"] == "sparse" for c in describe["classes"]) == sparse
