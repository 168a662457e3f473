"""Narrow cells, whose stencils have hundreds of cells: a few atoms each, at the
edges of the rule that cuts a group's stencil into runs; the oracle's list, bit
for bit."""

import numpy as np
import pytest

from helpers import assert_same

pytestmark = pytest.mark.gpu

PBC3 = [True, True, True]


@pytest.mark.parametrize("n,rc", [(1, 7.0), (1, 9.0), (2, 10.0), (8, 14.0), (16, 20.0), (33, 14.0),
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
    got = nl.build_neighborlists(nl.PyCell(h.tolist()), pos, rc)
    assert_same(got, oracle.search_single(pos, h, PBC3, rc, nthreads=8), "narrow cell")
