"""Bins of every size class on the builds that scatter atoms into sorted bins:
rank placement up to 512 atoms, one CTA's sort in shared memory up to 2048, its
merge path above -- for the pair tasks, several cutoffs (FP32 and FP64), and the
group search above the bucket build's atoms and bins; chunk boxes on dense grids.
The oracle's list, bit for bit."""

import numpy as np
import pytest

from helpers import assert_same

pytestmark = pytest.mark.gpu

PBC3 = [True, True, True]


@pytest.fixture(scope="module")
def nl():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import neighborlist_rs

    return neighborlist_rs


def clustered(n_gas, n_blob, box, seed):
    rng = np.random.default_rng(seed)
    pos = np.concatenate([rng.random((n_gas, 3)) * box,
                          0.5 * box + 0.3 + rng.random((n_blob, 3)) * 1.5])
    return pos[rng.permutation(len(pos))]


@pytest.mark.parametrize("n_blob", [500, 900, 2050, 4500])
@pytest.mark.parametrize("path", ["pair tasks", "two cutoffs", "five cutoffs"])
def test_large_bins_of_the_scattered_build(nl, oracle, path, n_blob):
    pos, h = clustered(3000, n_blob, 60.0, n_blob), np.eye(3) * 60.0
    cell = nl.PyCell(h.tolist())
    before = nl.set_single_pipeline(1)
    try:
        if path == "pair tasks":
            assert_same(nl.build_neighborlists(cell, pos, 5.0),
                        oracle.search_single(pos, h, PBC3, 5.0, nthreads=8), path)
            assert nl.last_single_pipeline() == 1
            return
        # (short cutoffs: the blob's pairs are counted, not all of them listed)
        cs = [0.2, 5.0] if path == "two cutoffs" else [0.1, 0.2, 0.3, 0.4, 5.0]
        got = nl.build_neighborlists_multi(cell, pos, cs)
        ref = oracle.search_single_multi(pos, h, PBC3, cs, nthreads=8)
        for q, rc in enumerate(cs):
            assert_same(got[q], ref[q], f"{path}, {rc}")
    finally:
        nl.set_single_pipeline(before)


@pytest.mark.parametrize("n_blob", [500, 900, 2500])
@pytest.mark.parametrize("n_gas,box", [(34000, 75.0), (34000, 120.0), (70000, 120.0), (3000, 80.0)])
def test_large_bins_of_the_group_search(nl, oracle, n_gas, box, n_blob):
    # 15^3 bins (k_prep's own scan), 24^3 (the scan over CTAs; one thread per
    # atom in the placement from 65,536 atoms), and few atoms in 16^3 bins
    pos, h = clustered(n_gas, n_blob, box, n_blob), np.eye(3) * box
    got = nl.build_neighborlists(nl.PyCell(h.tolist()), pos, 5.0)
    assert_same(got, oracle.search_single(pos, h, PBC3, 5.0, nthreads=8), "group search")
    assert nl.last_single_pipeline() == 0


def test_chunk_boxes_of_dense_grids(nl, oracle):
    # 3 bins per axis, some 740 atoms each
    pos, h = np.random.default_rng(11).random((20000, 3)) * 46.0, np.eye(3) * 46.0
    before = nl.set_single_pipeline(1)
    try:
        got = nl.build_neighborlists(nl.PyCell(h.tolist()), pos, 14.0)
    finally:
        nl.set_single_pipeline(before)
    assert_same(got, oracle.search_single(pos, h, PBC3, 14.0, nthreads=8), "pair tasks")
