"""The skin list's two launches: stored lists around the tile (2048 edges),
the warp's run (256) and the mask word (32), no stored edges at all, and one
manager updated on changing streams and threads without a synchronisation
between.  Whole numbers: equality with the oracle's filter."""

import threading

import numpy as np
import pytest

from helpers import assert_same

pytestmark = pytest.mark.gpu

PBC3 = [True, True, True]


@pytest.fixture(scope="module")
def torch():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


# a chain of atoms 1 apart, skin list of n - 1 edges, every third bond stretched
@pytest.mark.parametrize("n", [2, 3, 32, 33, 34, 257, 258, 2048, 2049, 2050, 4097])
def test_list_sizes(torch, oracle, n):
    import neighborlist_rs as nl
    from neighborlist_rs.verlet import VerletList

    pos = np.zeros((n, 3))
    pos[:, 0] = np.arange(n)
    rows = np.diag([n + 50.0, 50.0, 50.0])
    now = pos.copy()
    now[::3, 1] = 0.3
    stored = oracle.search_single(pos, rows, PBC3, 1.6, nthreads=8)
    assert stored[0].shape[1] == n - 1
    want = oracle.verlet_filter(now, rows, stored, 1.01)
    with VerletList(1.01, 0.61) as vl:
        cell = nl.PyCell(rows.tolist())
        vl.update(cell, torch.from_numpy(pos).cuda())
        for p in (torch.from_numpy(now).cuda(), now):
            res = vl.update(cell, p)
            assert not vl.rebuilt
            if p is not now:
                res = {k: v.cpu().numpy() for k, v in res.items()}
            assert_same(res, want, f"n {n}")


def test_streams_and_threads(torch, oracle):
    import neighborlist_rs as nl
    from neighborlist_rs.verlet import VerletList

    rng = np.random.default_rng(7)
    rows = np.eye(3) * 40.0
    pos = rng.random((6000, 3)) * 40.0
    cell = nl.PyCell(rows.tolist())
    stored = oracle.search_single(pos, rows, PBC3, 5.0, nthreads=8)
    moved = [pos + 0.1 * rng.random((6000, 3)) for _ in range(4)]
    wants = [oracle.verlet_filter(p, rows, stored, 4.0) for p in moved]
    dev = [torch.from_numpy(p).cuda() for p in moved]
    streams = [torch.cuda.default_stream(), torch.cuda.Stream(), torch.cuda.Stream()]
    got = []
    with VerletList(4.0, 1.0) as vl:
        vl.update(cell, torch.from_numpy(pos).cuda())
        torch.cuda.synchronize()

        def step(k):
            with torch.cuda.stream(streams[k % 3]):
                got.append((k % 4, vl.update(cell, dev[k % 4])))

        for k in range(24):
            if k % 5 == 4:
                t = threading.Thread(target=step, args=(k,))
                t.start()
                t.join()
            else:
                step(k)
        assert vl.rebuilt is False
    torch.cuda.synchronize()
    for k, res in got:
        assert_same({a: v.cpu().numpy() for a, v in res.items()}, wants[k], f"positions {k}")
