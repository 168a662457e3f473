"""The skin list's packed form: stored edges whose image shifts fit ten bits
and ones that do not (atoms hundreds of cells away), lists around the
compaction's tile of 2048 stored edges, an empty list, and systems of
changing size through one manager.  Whole numbers: equality with the oracle's
filter of the oracle's list."""

import numpy as np
import pytest

from helpers import assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("far", [0, 900])
def test_packed_list_matches_oracle(oracle, far):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import neighborlist_rs as nl
    from neighborlist_rs.verlet import VerletList

    rng = np.random.default_rng(31)
    rc, skin = 3.0, 0.8
    with VerletList(rc, skin) as vl:
        for n in (1, 170, 175, 180, 1500, 3100, 40):
            edge = (n / 0.05) ** (1.0 / 3.0) + 4.0
            h = np.array([[edge, 0.0, 0.0], [0.1 * edge, edge, 0.0], [0.0, -0.1 * edge, edge]]).T
            pos = rng.random((n, 3)) @ h.T
            pos = pos + rng.integers(-far, far + 1, (n, 3)) @ h.T
            cell = nl.PyCell(h.tolist())
            stored = oracle.search_single(pos, h, [True] * 3, rc + skin, nthreads=8)
            for k, by in enumerate((0.0, 0.1, 0.2)):
                now = pos + by * (rng.random((n, 3)) - 0.5)
                res = vl.update(cell, pos if k == 0 else now)
                assert vl.rebuilt == (k == 0)
                want = oracle.verlet_filter(pos if k == 0 else now, h, stored, rc)
                assert_same(res, want, f"n {n} far {far} step {k}")
