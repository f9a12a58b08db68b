"""The dense path keeps the rate that its Prim loop allows, whatever the hierarchy code beside it needs."""

import json

import numpy as np
import pytest

from tests.test_gpu_cluster import forced_variant

pytestmark = pytest.mark.gpu


def _dense_plan(sizes, dims, ms):
    from hdbscan_gb300 import _lib
    from hdbscan_gb300._cuda import Plan

    offsets = np.concatenate([[0], np.cumsum(sizes)])
    return Plan(offsets, dims, min_samples=ms, precision="float32", test_flags=_lib.HDB_FLAG_NO_SPARSE)


def _milliseconds(plan, X):
    import torch

    workspace = plan.workspace()
    times = []
    for _ in range(9):
        start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        start.record()
        plan.forward(X, workspace=workspace)
        end.record()
        end.synchronize()
        times.append(start.elapsed_time(end))
    return float(np.median(times[2:]))


def test_eight_slots_with_core_distances(cuda):
    # A step with core distances reads one more word a slot than one without: the same rate within a quarter.
    # (Row reads one after the other took twice the time.)
    import torch

    X = torch.randn(4001, 16, device=cuda)
    with forced_variant("float32", 512, 8, 0, 1):
        unit, cores = (_milliseconds(_dense_plan([4001], 16, ms), X) for ms in (2, 10))
    assert cores < 1.25 * unit


# (threads, dims of the variant, points, dims, CTAs an SM)
@pytest.mark.parametrize("threads, register, n, dims, ctas", [
    (256, 0, 300, 64, 3), (128, 8, 130, 4, 4), (128, 0, 200, 64, 4), (64, 0, 100, 64, 4), (64, 8, 100, 4, 4)])
def test_windows_an_sm_holds(cuda, threads, register, n, dims, ctas):
    # As many CTAs an SM as the Prim loop's registers allow, in batches that fill them.
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    with forced_variant("float32", threads, 2, register, 1, small=True):
        plan = _dense_plan([n] * (4 * sms * ctas), dims, 2)  # (matrix classes are cut into four chunks)
        classes = json.loads(plan.describe())["classes"]
    assert classes and all(c["threads"] == threads and c["register_dims"] == register for c in classes)
    assert all(c["grid"] >= sms * ctas for c in classes)
