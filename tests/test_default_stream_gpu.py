"""The torch entry points on torch's default stream follow the work queued on
it: positions whose values are still being computed when the call is made, a
tensor that is overwritten right after it, and results consumed without a
synchronisation.  Whole numbers: equality with the oracle."""

import numpy as np
import pytest

from helpers import assert_same

pytestmark = pytest.mark.gpu

PBC3 = [True, True, True]


@pytest.mark.parametrize("n", [300, 4000])
@pytest.mark.parametrize("side_stream", [False, True])
def test_calls_follow_the_current_stream(oracle, n, side_stream):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import neighborlist_rs as nl
    from neighborlist_rs.verlet import VerletList

    rng = np.random.default_rng(n)
    edge = (n / 0.1) ** (1.0 / 3.0)
    pos = rng.random((n, 3)) * edge
    moved = pos + 0.05 * (rng.random((n, 3)) - 0.5)
    rows = np.eye(3) * edge
    cell = nl.PyCell(rows.tolist())
    ref = oracle.search_single(moved, rows, PBC3, 4.0, nthreads=8)
    stored = oracle.search_single(pos, rows, PBC3, 5.0, nthreads=8)
    want = oracle.verlet_filter(moved, rows, stored, 4.0)
    big = torch.ones((4096, 4096), device="cuda")
    target = torch.from_numpy(moved).cuda()
    stream = torch.cuda.Stream() if side_stream else torch.cuda.default_stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream), VerletList(4.0, 1.0) as vl:
        vl.update(cell, torch.from_numpy(pos).cuda())
        for _ in range(3):
            d = torch.from_numpy(pos).cuda()
            for _ in range(20):  # some milliseconds of work ahead of the positions
                big = (big @ big) * (1.0 / 4096.0)
            d.copy_(target)
            got = nl.build_neighborlists_torch(cell, d, 4.0)
            kept = vl.update(cell, d)
            assert not vl.rebuilt
            d.zero_()
            both = [{k: v.cpu().numpy() for k, v in r.items()} for r in (got, kept)]
            assert_same(both[0], ref, "build")
            assert_same(both[1], want, "skin list")
