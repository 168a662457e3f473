"""The group search's packed candidates: the image shifts' bits depend on the
number of atoms (a third of what the index leaves of 32), and a window with a
shift outside them reads the plain ones.  Atoms up to `far` cells away, around
the range's ends for each size.  Whole numbers: equality with the oracle."""

import numpy as np
import pytest

from helpers import assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,far", [(n, far) for n, half in ((600, 64), (1025, 64), (5000, 32),
                                                            (40000, 16))
                                   for far in (1, half - 3, half - 1, half, half + 1, 700)])
def test_shifts_around_the_packed_range(oracle, n, far):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import neighborlist_rs as nl

    rng = np.random.default_rng(n + far)
    edge = (n / 0.1) ** (1.0 / 3.0)
    rows = np.array([[edge, 0, 0], [0.1 * edge, edge, 0], [0, -0.1 * edge, edge]])
    away = rng.integers(-1, 2, (n, 3))
    away[rng.random(n) < 0.02] = [far, -far, far - 1]
    pos = rng.random((n, 3)) @ rows + away @ rows
    ref = oracle.search_single(pos, rows, [True] * 3, 3.5, nthreads=8)
    got = nl.build_neighborlists_torch(nl.PyCell(rows.tolist()), torch.from_numpy(pos).cuda(), 3.5)
    assert_same({k: v.cpu().numpy() for k, v in got.items()}, ref, f"n {n} far {far}")
