"""Several lists of a batch written from the count pass's records (up to four
lists; five take the recomputing pass): uneven systems of all three searches,
atoms with more records than one segment holds, and an arena that is grown.
Whole numbers: equality with the oracle."""

import numpy as np
import pytest

from helpers import assert_same

pytestmark = pytest.mark.gpu

PBC3 = [True, True, True]


def _systems(kind):
    from neighborlist_rs import workloads as W

    if kind == "uneven":  # half isolated, half in skewed cells
        return W.concat_batch(W.uneven_batch(n_systems=96, seed=61))
    rng = np.random.default_rng(62)
    pos, batch, cells = [], [], []
    for s, n in enumerate([1, 2, 31, 33, 65, 300] if kind == "tight" else [700, 5, 1200]):
        rows = np.diag(rng.uniform(4.0, 6.0, 3)) if kind == "tight" else np.zeros((3, 3))
        pos.append(rng.random((n, 3)) @ (rows if kind == "tight" else np.eye(3) * 16.0))
        batch.append(np.full(n, s, np.int32))
        cells.append(rows)
    return np.concatenate(pos), np.concatenate(batch), np.array(cells)


@pytest.mark.parametrize("disjoint", [False, True])
@pytest.mark.parametrize("kind,cutoffs", [
    ("uneven", [5.0, 3.0]),
    ("uneven", [2.0, 5.0, 3.5]),
    ("uneven", [2.0, 5.0, 3.5, 5.0]),
    ("uneven", [2.0, 5.0, 3.5, 0.5, 4.0]),
    ("tight", [7.0, 2.0, 4.0, 0.1]),
    ("dense", [6.0, 2.0]),
])
def test_lists_from_records(oracle, kind, cutoffs, disjoint):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import neighborlist_rs as nl

    pos, batch, cells = _systems(kind)
    ocells = [None if not c.any() else (c.T, PBC3) for c in cells]
    ref = oracle.search_batch(pos, batch, ocells, cutoffs, disjoint=disjoint, nthreads=16)
    for call in range(4):  # timed shapes, direct, captured, replayed
        got = nl.build_neighborlists_batch_multi(pos, batch, cells=cells, cutoffs=cutoffs,
                                                 disjoint=disjoint)
        for q, rc in enumerate(cutoffs):
            assert_same(got[q], ref[q], f"call {call} rc {rc}")
