"""The torch entry points return when the list's size is known; the last
kernels may still read the positions.  Positions of another stream, dropped
right after the call, are not handed out again before those are done."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [900, 200_000])  # brute force; group search, some 100 us of writing
@pytest.mark.parametrize("owner,user", [("default", "side"), ("side", "default"),
                                        ("side", "side 2")])
def test_dropped_positions_are_kept_until_they_are_read(n, owner, user):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import neighborlist_rs as nl

    stream = {"default": torch.cuda.default_stream(), "side": torch.cuda.Stream(),
              "side 2": torch.cuda.Stream()}
    edge = (n / 0.1) ** (1.0 / 3.0)
    pos = torch.from_numpy(np.random.default_rng(n).random((n, 3)) * edge).cuda()
    torch.cuda.synchronize()
    for _ in range(4):
        with torch.cuda.stream(stream[owner]):
            d = pos.clone()
        torch.cuda.synchronize()
        with torch.cuda.stream(stream[user]):
            r = nl.build_neighborlists_torch(None, d, 5.0, vectors=True, distances=True)
        del d
        with torch.cuda.stream(stream[owner]):
            again = torch.full_like(pos, 1e6)  # (the dropped tensor's memory, were it free)
        torch.cuda.synchronize()
        src, dst = r["edge_index"]
        assert torch.equal(r["vectors"], pos[dst] - pos[src])
        assert int(src.shape[0]) > 4 * n
        del again, r


def test_positions_that_require_grad():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import neighborlist_rs as nl

    pos = torch.rand((2000, 3), dtype=torch.float64, device="cuda") * 27.0
    want = nl.build_neighborlists_torch(None, pos, 4.0)
    torch.cuda.synchronize()
    p = pos.clone().requires_grad_(True)
    for s in (torch.cuda.default_stream(), torch.cuda.Stream()):
        torch.cuda.synchronize()
        with torch.cuda.stream(s):
            for q in (p, p * 1.0):
                got = nl.build_neighborlists_torch(None, q, 4.0)
                torch.cuda.synchronize()
                assert torch.equal(got["edge_index"], want["edge_index"])
                assert not got["edge_index"].requires_grad
