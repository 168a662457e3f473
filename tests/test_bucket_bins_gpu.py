"""The bucket build's bins at, just above and far above their buckets, and
systems of uneven density of several sizes in a row: the oracle's list, bit
for bit."""

import numpy as np
import pytest

from helpers import assert_same

pytestmark = pytest.mark.gpu

PBC3 = [True, True, True]
RC, BINS = 6.0, 14  # 14^3 bins: 16 MB hold 496 entries of 12 bytes for each


@pytest.fixture(scope="module")
def nl():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import neighborlist_rs

    return neighborlist_rs


@pytest.mark.parametrize("k", [495, 496, 497, 1500])
def test_one_bin_around_its_bucket(nl, oracle, k):
    rng = np.random.default_rng(k)
    n, box = 5000, RC * BINS + 0.5
    width = box / BINS
    pos = rng.random((n, 3)) * box
    inside = np.floor(pos / width).astype(int)
    pos[(inside == 7).all(axis=1)] = 0.25 * width  # (no other atom in the bin)
    pos[rng.permutation(n)[:k]] = (7.0 + 0.02 + 0.96 * rng.random((k, 3))) * width
    in_bin = (np.floor(pos / width).astype(int) == 7).all(axis=1)
    assert in_bin.sum() == k
    cell = nl.PyCell((np.eye(3) * box).tolist())
    got = nl.build_neighborlists(cell, pos, RC)
    assert_same(got, oracle.search_single(pos, np.eye(3) * box, PBC3, RC, nthreads=8), f"k {k}")


def test_uneven_density_of_several_sizes(nl, oracle):
    rng = np.random.default_rng(4)
    for n in (700, 5200, 2300, 9100, 1100, 5200, 12000):
        box = (n / 0.02) ** (1.0 / 3.0)
        pos = rng.random((n, 3)) * box
        pos[: n // 2] *= 0.35
        cell = nl.PyCell((np.eye(3) * box).tolist())
        ref = oracle.search_single(pos, np.eye(3) * box, PBC3, RC, nthreads=8)
        assert_same(nl.build_neighborlists(cell, pos, RC), ref, f"n {n}")
