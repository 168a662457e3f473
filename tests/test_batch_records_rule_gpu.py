"""Several lists of a batch without cells, on both sides of the rule that takes
records instead of testing again (112 atoms in an atom's system on average),
and of one with a single cell in it.  Whole numbers: equality with the oracle."""

import numpy as np
import pytest

from helpers import assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("disjoint", [False, True])
@pytest.mark.parametrize("n,one_cell", [(1, False), (112, False), (113, False), (40, True)])
@pytest.mark.parametrize("cutoffs", [[3.0, 5.0], [5.0, 2.0, 3.5, 5.0]])
def test_isolated_batches(oracle, n, one_cell, cutoffs, disjoint):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import neighborlist_rs as nl

    rng = np.random.default_rng(n)
    edge = 1.5 + (n / 0.1) ** (1.0 / 3.0)
    pos = rng.random((12 * n, 3)) * edge
    batch = np.repeat(np.arange(12, dtype=np.int32), n)
    cells = np.zeros((12, 3, 3))
    if one_cell:
        cells[7] = np.eye(3) * edge
    ocells = [None if not c.any() else (c, [True] * 3) for c in cells]
    ref = oracle.search_batch(pos, batch, ocells, cutoffs, disjoint=disjoint, nthreads=8)
    for call in range(3):  # direct, captured, replayed
        got = nl.build_neighborlists_batch_multi(pos, batch, cells=cells if one_cell else None,
                                                 cutoffs=cutoffs, disjoint=disjoint)
        for q, rc in enumerate(cutoffs):
            assert_same(got[q], ref[q], f"call {call} rc {rc}")
