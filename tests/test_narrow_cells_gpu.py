"""Narrow cells, whose stencils have hundreds of cells: a few atoms each, at the
edges of the rules that choose the pair tasks or the group search for them and
cut a group's stencil into runs; the oracle's list, bit for bit."""

import numpy as np
import pytest

from helpers import assert_same

pytestmark = pytest.mark.gpu

PBC3 = [True, True, True]


@pytest.mark.parametrize("n,rc", [(1, 7.0), (1, 9.0), (2, 10.0), (8, 14.0), (16, 20.0), (33, 14.0), (128, 25.0), (129, 25.0),
                                  (100, 25.0), (300, 25.0)])
@pytest.mark.parametrize("skewed", [False, True])
def test_few_atoms_many_images(oracle, n, rc, skewed):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import neighborlist_rs as nl

    rng = np.random.default_rng(n)
    edge = (n / 0.1) ** (1.0 / 3.0)
    h = np.eye(3) * edge
    if skewed:
        h = np.array([[1.0, 0.8, 0.7], [0.0, 0.6, 0.2], [0.0, 0.0, 0.68]]) * edge * 2.0 ** (1.0 / 3.0)
    pos = rng.random((n, 3)) @ h.T
    cell = nl.PyCell(h.tolist())
    ref = oracle.search_single(pos, h, PBC3, rc, nthreads=8)
    for call in range(3):  # direct, captured, replayed
        assert_same(nl.build_neighborlists(cell, pos, rc), ref, f"call {call}")
    cells = np.prod(2 * np.ceil(rc * np.linalg.norm(np.linalg.inv(h), axis=1)) + 1)
    if cells <= 1024:
        assert nl.last_single_pipeline() == (1 if n <= 128 and cells > 125 else 0)
    got = nl.build_neighborlists_ex(cell, pos, rc, vectors=True)  # (one pass with the options)
    assert_same(got, ref, "with vectors")
    assert np.array_equal(got["vectors"], oracle.edge_extras(pos, h, ref, directed=False)[2])
