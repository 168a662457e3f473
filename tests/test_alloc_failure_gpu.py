"""Workspace allocations that fail (the failure-detection hook, on the host):
whichever allocation it is, the call gives the exact list or reports that there
is no memory, and the next call on the same workspace is exact.  Each attempt
runs in a thread of its own, whose workspace starts empty."""

import ctypes
import threading

import numpy as np
import pytest

from helpers import assert_same

pytestmark = pytest.mark.gpu

PBC3 = [True, True, True]


@pytest.fixture(scope="module")
def nl():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import neighborlist_rs

    neighborlist_rs._lib.nlb_debug_fail_alloc.argtypes = [ctypes.c_int32, ctypes.c_int32]
    return neighborlist_rs


def in_thread(f):
    out = []

    def run():
        try:
            out.append(f())
        except BaseException as e:  # handed to the caller
            out.append(e)

    t = threading.Thread(target=run)
    t.start()
    t.join()
    if isinstance(out[0], BaseException):
        raise out[0]
    return out[0]


def system(kind):
    rng = np.random.default_rng(5)
    if kind == "isolated":
        return rng.random((3000, 3)) * 31.0, None, 4.0
    if kind == "blob":  # more edges than the mean density tells: the arrays are grown
        rows = np.eye(3) * 60.0
        return (np.concatenate([rng.random((1200, 3)) * 8.0, rng.random((1800, 3)) * 60.0]), rows,
                4.0)
    n, rc = {"brute": (700, 4.0), "bucket": (3000, 4.0), "bins": (12000, 2.0)}[kind]
    rows = np.eye(3) * (n / 0.1) ** (1.0 / 3.0)
    return rng.random((n, 3)) @ rows, rows, rc


@pytest.mark.parametrize("kind", ["brute", "bucket", "bins", "blob", "isolated"])
@pytest.mark.parametrize("entry", ["host", "vectors", "owned"])
def test_every_allocation_of_a_build(nl, oracle, kind, entry):
    import torch

    pos, rows, rc = system(kind)
    cell = None if rows is None else nl.PyCell(rows.tolist())
    ref = oracle.search_single(pos, rows, None if rows is None else PBC3, rc, nthreads=8)
    vec = oracle.edge_extras(pos, rows, ref, directed=True)[2]
    d_pos = torch.from_numpy(pos).cuda()
    torch.cuda.synchronize()

    def build():
        if entry == "host":
            return nl.build_neighborlists(cell, pos, rc)
        if entry == "owned":
            r = nl.build_neighborlists_torch(cell, d_pos, rc)
        else:
            r = nl.build_neighborlists_torch(cell, d_pos, rc, directed=True, vectors=True)
            assert np.array_equal(r["vectors"].cpu().numpy(), vec)
            m = ref[0].shape[1]
            r = {"edge_index": r["edge_index"][:, :m], "shift": r["shift"][:m]}
        return {k: v.cpu().numpy() for k, v in r.items()}

    def attempt(nth, count):
        assert nl._lib.nlb_debug_fail_alloc(nth, count) == 0
        try:
            assert_same(build(), ref, f"allocation {nth}")
            ok = True
        except RuntimeError as e:
            assert "alloc" in str(e)
            ok = False
        assert nl._lib.nlb_debug_fail_alloc(0, 0) == 0
        for call in range(3):  # the same workspace, all memory there
            assert_same(build(), ref, f"after allocation {nth}, call {call}")
        return ok

    tries = range(0, 52, 1 if entry == "host" else 3)
    passed = [in_thread(lambda: attempt(nth, 1)) for nth in tries]
    assert passed[-1]  # (no build allocates as often)
    # A search that does not find its memory is replaced by one that needs less;
    # nothing replaces the positions (host), the bounds (isolated, on the device)
    # and the options' own arrays of that other search.
    if kind != "brute":
        first = 1 if entry == "host" or kind == "isolated" else 0
        assert all(passed[first:])
    for nth in (0, 3, 12, 30):  # no memory at all from there on
        in_thread(lambda: attempt(nth, 1000))


def test_every_allocation_of_a_skin_list(nl, oracle):
    import torch

    from neighborlist_rs.verlet import VerletList

    rng = np.random.default_rng(6)
    systems = []
    for n in (400, 5000):
        rows = np.eye(3) * (n / 0.1) ** (1.0 / 3.0)
        pos = rng.random((n, 3)) @ rows
        moved = pos + 0.05 * (rng.random((n, 3)) - 0.5)
        stored = oracle.search_single(pos, rows, PBC3, 3.0, nthreads=8)
        systems.append((nl.PyCell(rows.tolist()), torch.from_numpy(pos).cuda(),
                        torch.from_numpy(moved).cuda(),
                        oracle.verlet_filter(pos, rows, stored, 2.0),
                        oracle.verlet_filter(moved, rows, stored, 2.0)))
    torch.cuda.synchronize()

    def check(vl, cell, pos, want, what):
        got = {k: v.cpu().numpy() for k, v in vl.update(cell, pos).items()}
        assert_same(got, want, what)

    def attempt(nth):
        with VerletList(2.0, 1.0) as vl:
            cell, pos, moved, first, later = systems[0]
            check(vl, cell, pos, first, "small")
            check(vl, cell, moved, later, "small, moved")
            cell, pos, moved, first, later = systems[1]  # (a larger one: everything grows)
            assert nl._lib.nlb_debug_fail_alloc(nth, 1) == 0
            try:
                check(vl, cell, pos, first, f"allocation {nth}")
            except RuntimeError as e:
                assert "alloc" in str(e)
            assert nl._lib.nlb_debug_fail_alloc(0, 0) == 0
            for call in range(2):
                check(vl, cell, pos, first, f"after allocation {nth}, call {call}")
                check(vl, cell, moved, later, f"after allocation {nth}, moved {call}")

    for nth in range(0, 60, 1):
        in_thread(lambda: attempt(nth))


def test_the_next_call_may_take_another_stream(nl, oracle):
    """A call that fails has waited for what it queued: the next one frees and
    writes the same workspace on another stream."""
    import torch

    sides = [torch.cuda.Stream() for _ in range(2)]
    systems = []
    for kind in ("brute", "bucket", "bins"):
        pos, rows, rc = system(kind)
        systems.append((nl.PyCell(rows.tolist()), torch.from_numpy(pos).cuda(), rc,
                        oracle.search_single(pos, rows, PBC3, rc, nthreads=8)))
    torch.cuda.synchronize()

    def attempt(nth):
        for k, (cell, pos, rc, ref) in enumerate(systems):  # (each larger: the workspace grows)
            assert nl._lib.nlb_debug_fail_alloc(nth, 1000) == 0
            with torch.cuda.stream(sides[k % 2]), pytest.raises(RuntimeError, match="alloc"):
                nl.build_neighborlists_torch(cell, pos, rc, vectors=True)
            assert nl._lib.nlb_debug_fail_alloc(0, 0) == 0
            with torch.cuda.stream(sides[(k + 1) % 2]):
                r = nl.build_neighborlists_torch(cell, pos, rc)
                assert_same({q: v.cpu().numpy() for q, v in r.items()}, ref, f"{nth}, {k}")

    for nth in (0, 1, 2, 3):
        in_thread(lambda: attempt(nth))
