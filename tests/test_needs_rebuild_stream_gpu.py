"""VerletList.needs_rebuild with a CUDA tensor follows the work queued on the
current torch stream, and refuses what update refuses."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side_stream", [False, True])
def test_needs_rebuild_follows_the_current_stream(side_stream):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import neighborlist_rs as nl
    from neighborlist_rs.verlet import VerletList

    n, edge = 4000, 34.2
    rng = np.random.default_rng(3)
    pos = torch.from_numpy(rng.random((n, 3)) * edge).cuda()
    step = torch.zeros_like(pos)
    step[17] = torch.tensor([0.75, 0.0, 1.0], dtype=torch.float64)  # length 1.25 > skin / 2
    cell = nl.PyCell((np.eye(3) * edge).tolist())
    big = torch.ones((4096, 4096), device="cuda")
    stream = torch.cuda.Stream() if side_stream else torch.cuda.default_stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream), VerletList(4.0, 1.0) as vl:
        vl.update(cell, pos)
        for _ in range(3):
            d = pos.clone()
            assert not vl.needs_rebuild(cell, d) and vl.max_displacement == 0.0
            for _ in range(20):  # some milliseconds of work ahead of the positions
                big = (big @ big) * (1.0 / 4096.0)
            d += step
            assert vl.needs_rebuild(cell, d)
            assert vl.max_displacement == pytest.approx(1.25, rel=1e-12)
            # (a tensor that is not contiguous, its copy queued the same way)
            t = d.t().contiguous().t()
            assert vl.needs_rebuild(cell, t) and not vl.needs_rebuild(cell, t - step)


def test_needs_rebuild_refuses_what_update_refuses():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from neighborlist_rs.verlet import VerletList

    good = torch.zeros((5, 3), dtype=torch.float64, device="cuda")
    with VerletList(4.0, 1.0) as vl:
        for bad in (good.float(), good.reshape(-1)):
            with pytest.raises(TypeError, match="float64"):
                vl.needs_rebuild(None, bad)
        with pytest.raises(ValueError, match=r"\(N, 3\)"):
            vl.needs_rebuild(None, torch.zeros((5, 4), dtype=torch.float64, device="cuda"))
        assert vl.needs_rebuild(None, good)  # no list yet
