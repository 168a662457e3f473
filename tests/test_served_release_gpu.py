"""DeviceResult.to_torch queues its copies on the current torch stream; a
release right after it does not hand the memory to the next requests before
the copies are done."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side_stream", [False, True])
@pytest.mark.parametrize("n", [300, 6000])  # a batched request and a large one
def test_release_right_after_to_torch(n, side_stream):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import neighborlist_rs as nl
    from neighborlist_rs.serving import Server

    rng = np.random.default_rng(n)
    edge = (n / 0.1) ** (1.0 / 3.0)
    cell = nl.PyCell((np.eye(3) * edge).tolist())
    pos = [rng.random((n, 3)) * edge for _ in range(8)]
    want = [nl.build_neighborlists(cell, p, 5.0) for p in pos]
    big = torch.ones((8192, 8192), device="cuda")
    stream = torch.cuda.Stream() if side_stream else torch.cuda.default_stream()
    torch.cuda.synchronize()
    with Server(hbm_budget_bytes=4 << 30, workers=2) as srv, torch.cuda.stream(stream):
        got = []
        for p in pos:
            r = srv.wait(srv.submit(cell, p, 5.0, device_result=True), timeout=60.0)
            for _ in range(2):  # some milliseconds of work ahead of the copies
                big = (big @ big) * (1.0 / 8192.0)
            got.append(r.to_torch())
            r.release()
        torch.cuda.synchronize()
        for k, (g, w) in enumerate(zip(got, want)):
            assert np.array_equal(g["edge_index"].cpu().numpy(), w["edge_index"]), k
            assert np.array_equal(g["shift"].cpu().numpy(), w["shift"]), k
        assert srv.stats()["reserved_bytes"] == 0
