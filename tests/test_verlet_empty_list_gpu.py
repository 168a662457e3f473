"""A skin list whose rebuild finds no edges: when the update returns, the
reference positions are stored -- the caller may overwrite its own, and the
next call may come on another stream."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [100, 200])  # a million and eight million atoms, none in reach
@pytest.mark.parametrize("entry", ["device", "host"])
def test_reference_is_stored_when_the_update_returns(side, entry):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import neighborlist_rs as nl
    from neighborlist_rs.verlet import VerletList

    g = torch.arange(side, dtype=torch.float64, device="cuda") * 2.0 + 1.0
    pos = torch.stack(torch.meshgrid(g, g, g, indexing="ij"), dim=-1).reshape(-1, 3).contiguous()
    kept = pos.clone()
    cell = nl.PyCell((np.eye(3) * 2.0 * side).tolist())
    h, pb = nl._cell_args(cell)
    n = pos.shape[0]
    flag = ctypes.c_int(0)
    host = pos.cpu().pin_memory().numpy() if entry == "host" else None
    side_stream = torch.cuda.Stream()
    first = torch.cuda.Stream(priority=-1)  # (its work runs ahead of copies still going)
    torch.cuda.synchronize()
    with VerletList(1.0, 0.5) as vl:
        for _ in range(3):
            if entry == "device":  # on the library's own stream
                out = nl._DevResult()
                some = pos[::1000]
                with torch.cuda.stream(first):
                    code = nl._lib.nlb_verlet_update_device(
                        vl._handle(), pos.data_ptr(), n, h, pb, ctypes.byref(flag),
                        ctypes.byref(out))
                    some.zero_()
                nl._check(code)
                m = int(out.n_edges)
            else:
                m = vl.update(cell, host)["edge_index"].shape[1]
                flag.value = int(vl.rebuilt)
                host[:] = 0.0
            assert m == 0 and flag.value == 1
            needs, disp = ctypes.c_int(-1), ctypes.c_double(-1.0)
            nl.set_stream(side_stream.cuda_stream)
            try:
                nl._check(nl._lib.nlb_verlet_needs_rebuild(
                    vl._handle(), ctypes.c_void_p(kept.data_ptr()), n, h, pb, 1,
                    ctypes.byref(needs), ctypes.byref(disp)))
            finally:
                nl.set_stream(None)
            assert disp.value == 0.0 and needs.value == 0
            torch.cuda.synchronize()
            moved = kept + 1.0  # the next update rebuilds
            pos.copy_(moved)
            if host is not None:
                host[:] = moved.cpu().numpy()
            kept = moved
            torch.cuda.synchronize()
