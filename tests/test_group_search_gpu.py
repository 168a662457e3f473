"""The two-launch group search against the oracle where its splits and
buffers have edges: bins of 31 to 33, 64, 65 and 513 atoms (groups of 32,
half-empty last groups, the placement's large bins), stencils of more than 32
cells (several describing rounds) and of one cell per segment, grids above
65,536 bins, shifts that do not fit the packed 10 bits, positions so far out
that wrapping loses bits (every hit rechecked), far fewer records and edges
expected than there are (both arrays grown), and sizes on both sides of the
segment rule.  Results are whole numbers: equality, no tolerance."""

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


def filled_bins(counts, rng, edge=4.0):
    """Bins of the given numbers of atoms in a row of cubes (one per bin)."""
    pos = [np.array([edge * b, 0.0, 0.0]) + edge * (0.02 + 0.96 * rng.random((k, 3)))
           for b, k in enumerate(counts)]
    return np.concatenate(pos), np.diag([edge * len(counts), edge, edge])


def case(name):
    rng = np.random.default_rng(97)
    if name == "group edges":
        pos, rows = filled_bins([31, 32, 33, 64, 65, 1, 0, 513, 40, 300], rng)
        return pos, rows, 4.0
    if name == "125 cells":
        rows = np.diag([6.0, 6.5, 7.0])
        return rng.random((1003, 3)) @ rows, rows, 7.5
    if name == "slab":  # 3 x 3 x 7 cells
        rows = np.diag([40.0, 41.0, 5.0])
        return rng.random((1501, 3)) @ rows, rows, 13.0
    if name == "many bins":
        rows = np.eye(3) * 200.0
        return rng.random((20_011, 3)) @ rows, rows, 4.8
    if name == "wide shifts":
        rows = np.array([[20.0, 0, 0], [3.0, 21.0, 0], [-2.0, 4.0, 22.0]])
        pos = rng.random((1200, 3)) @ rows
        return pos + rng.integers(-900, 900, (1200, 3)) @ rows, rows, 5.0
    if name == "far out":
        rows = np.eye(3) * 20.0
        return rng.random((1100, 3)) * 20.0 + 3.0e11, rows, 5.0
    if name == "clustered":
        rows = np.eye(3) * 90.0
        pos = np.concatenate([rng.random((5000, 3)) * 9.0 + 40.0, rng.random((700, 3)) * 90.0])
        return pos, rows, 4.5
    n = int(name)
    rows = np.eye(3) * (n / 0.1) ** (1.0 / 3.0)
    return rng.random((n, 3)) @ rows, rows, 6.0


@pytest.mark.parametrize("name", ["group edges", "125 cells", "slab", "many bins", "wide shifts",
                                  "far out", "clustered", "1000", "4097", "70001", "140003"])
def test_group_search_matches_oracle(nl, oracle, name):
    import torch

    pos, rows, rc = case(name)
    cell = nl.PyCell(rows.T.tolist())
    ref = oracle.search_single(pos, rows.T, PBC3, rc, nthreads=16)
    d = torch.from_numpy(np.ascontiguousarray(pos)).cuda()
    for k in range(2):
        got = nl.build_neighborlists_torch(cell, d, rc)
        assert nl.last_single_pipeline() == 0
        assert_same({"edge_index": got["edge_index"].cpu().numpy(),
                     "shift": got["shift"].cpu().numpy()}, ref, f"{name} device #{k}")
    assert_same(nl.build_neighborlists(cell, pos, rc), ref, f"{name} host")
