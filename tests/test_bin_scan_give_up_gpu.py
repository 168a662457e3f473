"""A bounded wait that runs out in the scan of the bins (grids above 4096
bins: several tiles): the build reports the error, no later kernel uses the
bin starts, and the next builds on the same workspace are exact.  One tile
withholds its publication (the failure-detection hook); nothing faults."""

import ctypes

import numpy as np
import pytest

from helpers import assert_same

pytestmark = pytest.mark.gpu

PBC3 = [True, True, True]
N, BOX, RC = 15000, 60.0, 3.0  # 20^3 bins: four tiles of 2048


@pytest.mark.parametrize("tile", [0, 1, 2])
@pytest.mark.parametrize("path", ["group", "group vectors", "pair tasks", "two cutoffs",
                                  "five cutoffs (FP64)", "no allocation"])
def test_bin_scan_gives_up_and_recovers(oracle, path, tile):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import neighborlist_rs as nl

    nl._lib.nlb_debug_scan_stall.argtypes = [ctypes.c_int32, ctypes.c_int32]
    rng = np.random.default_rng(17)
    rows = np.eye(3) * BOX
    pos = rng.random((N, 3)) * BOX
    cell = nl.PyCell(rows.tolist())
    ref = oracle.search_single(pos, rows, PBC3, RC, nthreads=8)
    d_pos = torch.from_numpy(pos).cuda()
    torch.cuda.synchronize()

    def noalloc():
        h9 = np.ascontiguousarray(rows.reshape(9))
        cap = ref[0].shape[1]
        ei = torch.zeros((2, cap), dtype=torch.int64, device="cuda")
        sh = torch.zeros((cap, 3), dtype=torch.int32, device="cuda")
        m = ctypes.c_int64(-1)
        torch.cuda.synchronize()
        nl._check(nl._lib.nlb_build_noalloc(
            ctypes.c_void_p(d_pos.data_ptr()), ctypes.c_int64(N), ctypes.c_double(RC),
            h9.ctypes.data_as(nl._dp), (ctypes.c_uint8 * 3)(1, 1, 1),
            ctypes.c_void_p(ei.data_ptr()), ctypes.c_void_p(sh.data_ptr()), ctypes.c_int64(cap),
            ctypes.byref(m), None))
        return {"edge_index": ei.cpu().numpy(), "shift": sh.cpu().numpy()}

    def torch_vectors():
        r = nl.build_neighborlists_torch(cell, d_pos, RC, vectors=True)
        return {k: r[k].cpu().numpy() for k in ("edge_index", "shift")}

    run = {
        "group": lambda: nl.build_neighborlists(cell, pos, RC),
        "group vectors": torch_vectors,
        "pair tasks": lambda: nl.build_neighborlists(cell, pos, RC),
        "two cutoffs": lambda: nl.build_neighborlists_multi(cell, pos, [2.0, RC])[1],
        "five cutoffs (FP64)": lambda: nl.build_neighborlists_multi(
            cell, pos, [1.0, 1.5, 2.0, 2.5, RC])[4],
        "no allocation": noalloc,
    }[path]
    before = nl.set_single_pipeline(1 if path == "pair tasks" else 0)
    try:
        for _ in range(2):
            assert nl._lib.nlb_debug_scan_stall(tile, 2048) == 0
            with pytest.raises(RuntimeError, match="prefix scan gave up waiting for a tile"):
                run()
            for k in range(3):
                assert_same(run(), ref, f"after, call {k}")
    finally:
        nl.set_single_pipeline(before)


def test_a_tile_past_the_bin_scan_is_left_for_the_search(oracle):
    """The bin scan takes the hook only for a tile that another one waits for;
    the group search's own scan takes it otherwise."""
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import neighborlist_rs as nl

    nl._lib.nlb_debug_scan_stall.argtypes = [ctypes.c_int32, ctypes.c_int32]
    rng = np.random.default_rng(18)
    rows = np.eye(3) * BOX
    pos = rng.random((N, 3)) * BOX
    cell = nl.PyCell(rows.tolist())
    ref = oracle.search_single(pos, rows, PBC3, RC, nthreads=8)
    for tile in (3, 40):  # the bin scan's last tile (nobody waits for it), and none of its tiles
        assert nl._lib.nlb_debug_scan_stall(tile, 2048) == 0
        with pytest.raises(RuntimeError, match="prefix scan gave up waiting for a tile"):
            nl.build_neighborlists(cell, pos, RC)
        assert_same(nl.build_neighborlists(cell, pos, RC), ref, "after")
