"""Brute force of one small system in two launches (one mask word per 32
candidates) and the auto-box bounds taken by several CTAs, against the oracle:
sizes around the warp and the 32-word limit, raw and minimum-image distances,
mixed periodicity, more edges than the density suggests, and isolated systems
around the bounds' CTA share.  Whole numbers: equality."""

import numpy as np
import pytest

from helpers import assert_same

pytestmark = pytest.mark.gpu


@pytest.fixture()
def nl():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import neighborlist_rs

    yield neighborlist_rs
    neighborlist_rs.set_brute_force_threshold(1000)


def both(nl, cell, pos, rc):
    import torch

    host = nl.build_neighborlists(cell, pos, rc)
    dev = nl.build_neighborlists_torch(cell, torch.from_numpy(pos).cuda(), rc)
    return host, {k: v.cpu().numpy() for k, v in dev.items()}


@pytest.mark.parametrize("pbc", [None, (True, True, True), (True, False, True)])
@pytest.mark.parametrize("n", [1, 2, 31, 33, 64, 65, 999, 1024, 1025])
def test_brute_rows_match_oracle(nl, oracle, n, pbc):
    rng = np.random.default_rng(n)
    nl.set_brute_force_threshold(2000)
    # (atoms crowded into an eighth of the box: several times the uniform edges)
    pos = np.ascontiguousarray(rng.random((n, 3)) * 13.0 + rng.integers(-1, 2, (n, 3)) * 26.0)
    h = np.eye(3) * 26.0
    h[0, 1] = 2.0
    cell = None if pbc is None else nl.PyCell(h.tolist(), pbc)
    oracle.set_thresholds(brute_force=2000)
    try:
        ref = oracle.search_single(pos, None if pbc is None else h, pbc, 4.0, nthreads=8)
    finally:
        oracle.set_thresholds()
    for what, got in zip(("host", "device"), both(nl, cell, pos, 4.0)):
        assert_same(got, ref, f"n {n} pbc {pbc} {what}")


@pytest.mark.parametrize("n", [1500, 4096, 4097, 70_003])
def test_isolated_bounds_match_oracle(nl, oracle, n):
    rng = np.random.default_rng(n)
    pos = rng.normal(size=(n, 3)) * (n / 0.3) ** (1.0 / 3.0) - 40.0
    ref = oracle.search_single(pos, None, None, 3.0, nthreads=16)
    for what, got in zip(("host", "device"), both(nl, None, pos, 3.0)):
        assert_same(got, ref, f"n {n} {what}")
