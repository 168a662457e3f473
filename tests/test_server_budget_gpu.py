"""A large request whose cell list and result fit the server's budget runs there,
also when the search's own workspace on top of them does not, and its whole
reservation is given back.  Whole numbers: equality with the oracle."""

import numpy as np
import pytest

from helpers import assert_same

pytestmark = pytest.mark.gpu


def test_budget_between_the_two_estimates(oracle):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import neighborlist_rs as nl
    from neighborlist_rs.serving import Server

    n, rc = 20000, 6.0
    rng = np.random.default_rng(8)
    edge = (n / 0.1) ** (1.0 / 3.0)
    rows = np.eye(3) * edge
    cell = nl.PyCell(rows.tolist())
    # positions, cell list and result at the mean density; the search's
    # records come to some 0.8 kB an atom more
    base = 28.0 * 1.3 * n * (0.05 * 4.0 / 3.0 * np.pi * rc ** 3 + 1.0) + 568.0 * n
    pos = [rng.random((n, 3)) * edge for _ in range(4)]
    with Server(hbm_budget_bytes=int(base * 1.02) + 4096, workers=2) as srv:
        tickets = [srv.submit(cell, p, rc) for p in pos]
        for t, p in zip(tickets, pos):
            assert_same(srv.wait(t, timeout=60.0),
                        oracle.search_single(p, rows, [True] * 3, rc, nthreads=8), "served")
        assert srv.stats()["reserved_bytes"] == 0
    with Server(hbm_budget_bytes=int(base * 0.98), workers=1) as srv:
        with pytest.raises(ValueError, match="budget"):
            srv.submit(cell, pos[0], rc)
