"""Repeated builds with output options are replayed as a graph; a build of the
same size whose cell has the matrix of an earlier call's auto-box is another
one, since only it adds H S to the vectors.  Whole numbers and floats: bit for
bit the oracle's."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N, RC = 1500, 3.0
SPAN = 24.0                        # exact, so that the auto-box's edges are too
BOX = SPAN + 2.0 * (RC + 1.0)


def _check(oracle, got, pos, h, pbc):
    half = oracle.search_single(pos, h, pbc, RC, nthreads=8)
    ei, sh, vec, dist = oracle.edge_extras(pos, h, half, directed=False)
    assert np.array_equal(got["edge_index"], ei) and np.array_equal(got["shift"], sh)
    assert np.array_equal(got["vectors"].view(np.int64), vec.view(np.int64))
    assert np.array_equal(got["distances"].view(np.int64), dist.view(np.int64))
    return half


@pytest.mark.parametrize("entry", ["host", "side stream"])
@pytest.mark.parametrize("auto_box_first", [True, False])
def test_auto_box_and_cell_of_one_matrix(oracle, entry, auto_box_first):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import neighborlist_rs as nl

    rng = np.random.default_rng(11)
    free = rng.random((N, 3)) * SPAN
    free[0], free[1] = 0.0, SPAN
    full = rng.random((N, 3)) * BOX
    h = np.eye(3) * BOX
    cell = nl.PyCell(h.tolist())
    stream = torch.cuda.Stream()
    buf = torch.empty((N, 3), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()

    def build(c, pos):
        if entry == "host":
            return nl.build_neighborlists_ex(c, pos, RC, vectors=True, distances=True)
        with torch.cuda.stream(stream):
            buf.copy_(torch.from_numpy(pos))
            r = nl.build_neighborlists_torch(c, buf, RC, vectors=True, distances=True)
            return {k: v.cpu().numpy() for k, v in r.items()}

    calls = [(None, free, None, None), (cell, full, h, [True] * 3)]
    if not auto_box_first:
        calls.reverse()
    crossing = 0
    for c, pos, hh, pbc in calls:
        for _ in range(4):  # direct, captured, replayed
            half = _check(oracle, build(c, pos), pos, hh, pbc)
        crossing += int((half[1] != 0).any(axis=1).sum())
    assert crossing > 100
