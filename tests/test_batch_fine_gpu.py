"""Batches too small to fill the GPU, which are cut into pieces of 16 to 128
atoms of any of their systems: sizes at the edges of the pieces, one system
and many, and batches on both sides of the rule (atoms and systems).  Whole
numbers: equality with the oracle."""

import numpy as np
import pytest

from helpers import assert_same

pytestmark = pytest.mark.gpu

PBC3 = [True, True, True]


@pytest.mark.parametrize("sizes,cutoffs", [
    ([1], [5.0]),
    ([15, 16, 17, 1, 33], [5.0, 3.0]),
    ([2048], [5.0]),
    ([31, 32, 33, 64, 65, 127, 128, 129, 700, 1025], [4.0]),  # pieces of 32
    ([1500] * 4 + [40], [4.0, 6.0]),  # of 64
    ([2047] * 5 + [100] * 60, [4.0]),  # of 128
    ([2000] * 9 + [900], [4.0]),  # just below the most atoms
    ([2000] * 9 + [1000], [4.0]),  # just above
    ([20] * 185, [4.0]),  # the most systems
    ([20] * 186, [4.0, 2.0, 3.0]),  # one more
])
def test_small_batches(oracle, sizes, cutoffs):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import neighborlist_rs as nl

    rng = np.random.default_rng(len(sizes))
    pos, batch, cells = [], [], []
    for s, n in enumerate(sizes):
        edge = (n / 0.1) ** (1.0 / 3.0)
        rows = np.array([[edge, 0, 0], [0.2 * edge, edge, 0], [0, -0.1 * edge, edge]])
        pos.append(rng.random((n, 3)) @ rows)
        batch.append(np.full(n, s, np.int32))
        cells.append(rows if s % 3 else np.zeros((3, 3)))
    pos, batch, cells = np.concatenate(pos), np.concatenate(batch), np.array(cells)
    ocells = [None if not c.any() else (c.T, PBC3) for c in cells]
    ref = oracle.search_batch(pos, batch, ocells, cutoffs, nthreads=16)
    for call in range(3):  # direct, captured, replayed
        got = nl.build_neighborlists_batch_multi(pos, batch, cells=cells, cutoffs=cutoffs)
        for q, rc in enumerate(cutoffs):
            assert_same(got[q], ref[q], f"call {call} rc {rc}")
