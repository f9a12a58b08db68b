"""The shares of the products' error bound (sparse_eta and sparse_chain in hdb_sparse.cuh), restated here, against
NumPy emulations of the arithmetic that they bound, on data that makes each share large."""

import re
from pathlib import Path

import numpy as np
import pytest

SOURCE = (Path(__file__).resolve().parents[1] / "hdbscan_gb300" / "csrc" / "hdb_sparse.cuh").read_text()


def eta(dims, low, rest):
    """low, rest: largest |lo|^2 / norm and |rest|^2 / norm of the points."""
    return 1.1 * (low + 2 * np.sqrt(rest) + 6 * 2.0**-20 + (dims // 8 + 32) * 2.0**-24)


def chain(dims):
    return 1.05 * (dims + 8) * 2.0**-24


def test_restated_formulas():
    assert re.search(r"return 1\.1f \* \(split \+ 6\.0f \* 9\.5367432e-7f \+ \(float\)\(a\.D / 8 \+ 32\) \* 5\.9604645e-8f\);",
                     SOURCE)
    assert re.search(r"split = __uint_as_float\(a\.split_share\[w\]\) \+ 2\.0f \* sqrtf\(", SOURCE)
    assert re.search(r"1\.05f \* \(float\)\(D \+ 8\) \* 5\.9604645e-8f : 0\.0f;", SOURCE)


def pairs(kind, dims, count, rng):
    """float32 points a, b [count, dims]."""
    if kind == "antipodal":
        a = np.abs(rng.normal(1, 0.01, (count, 1))) * np.ones(dims)
        return a.astype(np.float32), -a.astype(np.float32)
    if kind == "half units":  # every coordinate after the first is rounded away, or up to a whole unit
        a = np.zeros((count, dims))
        a[:, 0] = 2.0
        a[:, 1:] = np.sqrt(2.0**-22) * (1 + np.linspace(-0.01, 0.01, count))[:, None]
        return a.astype(np.float32), np.zeros((count, dims), np.float32)
    if kind == "increments":
        a = np.cumsum(rng.uniform(0, 1e-3, (count, dims)), axis=1)
        return a.astype(np.float32), np.zeros((count, dims), np.float32)
    a = rng.normal(0, 1, (count, dims))
    return a.astype(np.float32), (a + rng.normal(0, 10.0 ** rng.uniform(-4, 1, (count, 1)), (count, dims))).astype(np.float32)


KINDS = ("antipodal", "half units", "increments", "normal")


@pytest.mark.parametrize("dims", [32, 100, 768, 2048])
@pytest.mark.parametrize("kind", KINDS)
def test_chain_covers_the_serial_float32_sum(kind, dims):
    a, b = pairs(kind, dims, 400, np.random.default_rng(dims))
    total = np.zeros(len(a), np.float32)
    for k in range(dims):
        delta = a[:, k] - b[:, k]
        total = total + delta * delta
    got = np.sqrt(total).astype(np.float64) ** 2
    true = np.sum((a.astype(np.float64) - b) ** 2, axis=1)
    error = np.abs(got - true)
    assert (error <= chain(dims) * true).all()
    if kind == "half units":  # the share is needed: no small fraction of it would do
        assert (error / true).max() > 0.2 * chain(dims)


def bfloat16(x):
    bits = x.astype(np.float32).view(np.uint32)
    return ((bits + 0x7FFF + ((bits >> 16) & 1)) & 0xFFFF0000).astype(np.uint32).view(np.float32)


@pytest.mark.parametrize("dims", [32, 100, 768, 2048])
@pytest.mark.parametrize("kind", KINDS)
def test_eta_covers_the_products(kind, dims):
    a, b = pairs(kind, dims, 400, np.random.default_rng(dims))
    centre = ((a[0] + b[0]) * np.float32(0.5)).astype(np.float32)
    za, zb = (a - centre).astype(np.float32), (b - centre).astype(np.float32)
    norms, parts, low, rest = [], [], 0.0, 0.0
    for z in (za, zb):
        high = bfloat16(z)
        low_part = bfloat16(z - high)
        parts.append((high, low_part))
        lanes = np.zeros((len(z), 32), np.float32)  # a warp's fused sums, then five additions
        for k in range(dims):
            lanes[:, k % 32] = (lanes[:, k % 32] + z[:, k].astype(np.float64) ** 2).astype(np.float32)
        while lanes.shape[1] > 1:
            half = lanes.shape[1] // 2
            lanes = lanes[:, :half] + lanes[:, half:]
        norms.append(lanes[:, 0])
        some = lanes[:, 0] > 0
        low = max(low, (np.sum(low_part.astype(np.float64) ** 2, axis=1)[some] / lanes[some, 0]).max())
        rest = max(rest, (np.sum((z - high - low_part).astype(np.float64) ** 2, axis=1)[some] / lanes[some, 0]).max())
    (ah, al), (bh, bl) = parts
    product = np.zeros(len(a), np.float32)
    for k in range(0, dims, 32):  # an accumulator of its own every 32 coordinates, then a float32 sum
        part = np.zeros(len(a), np.float32)
        for x, y in ((ah, bl), (al, bh), (ah, bh)):
            for h in range(k, min(k + 32, dims), 16):
                step = np.sum(x[:, h:h + 16].astype(np.float64) * y[:, h:h + 16], axis=1)
                part = (part + step).astype(np.float32)
        product = product + part
    got = (norms[0] + norms[1]).astype(np.float64) - 2.0 * product
    true = np.sum((a.astype(np.float64) - b) ** 2, axis=1)
    both = np.sum(za.astype(np.float64) ** 2, axis=1) + np.sum(zb.astype(np.float64) ** 2, axis=1)
    assert (np.abs(got - true) <= eta(dims, low, rest) * both).all()
    if kind == "antipodal":  # rounding of one sign in all coordinates: more than it averages to, up to 2^-15
        assert (np.abs(got - true) / both).max() > 2 * 3 * 2.0**-18
    assert low <= 2.0**-16 and rest <= 2.0**-34
