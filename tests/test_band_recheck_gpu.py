"""Pairs within the FP32 test's guard band, many to a chunk: lattices whose
cutoff is one of their distances, cells as wide as the cutoff, and positions so
far from the cell that certain hits are rechecked too.  The oracle's list, bit
for bit."""

import numpy as np
import pytest

from helpers import assert_same

pytestmark = pytest.mark.gpu

PBC3 = [True, True, True]


def fcc(k, a):
    g = np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 1, 3)
    basis = np.array([[0, 0, 0], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]])
    return (g + basis).reshape(-1, 3) * a + 0.1, np.eye(3) * a * k


def systems():
    rng = np.random.default_rng(9)
    for k in (1, 2, 3, 10):
        for rc in (8.0, np.sqrt(2.0) * 4.0, np.nextafter(8.0, 9.0)):
            yield f"fcc {4 * k ** 3}, rc {rc}", *fcc(k, 4.0), rc
    for n in (1, 31, 33, 100):  # every atom and its image at the cutoff
        yield f"{n} atoms, rc = edge", rng.random((n, 3)) * 10.0, np.eye(3) * 10.0, 10.0
    pos, h = fcc(6, 4.0)
    yield "fcc, shuffled and moved by cells", (pos + rng.integers(-2, 3, pos.shape) * 24.0)[
        rng.permutation(len(pos))], h, 8.0
    yield "far from the cell", pos + 1e12, h, 8.0


def test_many_pairs_in_the_guard_band(oracle):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import neighborlist_rs as nl

    for what, pos, h, rc in systems():
        got = nl.build_neighborlists(nl.PyCell(h.tolist()), pos, rc)
        assert_same(got, oracle.search_single(pos, h, PBC3, rc, nthreads=8), what)
