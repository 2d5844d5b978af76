"""The scratch a context keeps between calls (tsg_scratch_bytes) is given back
when device memory runs out: to any other call of any context on the device,
and a product that has no room beside it, or for the row path's tables, is run
once more without both.  The device is not filled for it: an allocation is told
that it is (tsg_inject_alloc_failure, kind 2)."""
import threading

import numpy as np
import pytest

from oracle import oracle as O
from test_rows_gpu import _cases, _rows

pytestmark = pytest.mark.gpu


@pytest.fixture()
def full(built_lib):
    """full(k): the k-th device allocation from now finds the memory full."""
    from tilespgemm_gb300 import _abi
    L = _abi.lib()
    yield lambda k: _abi.check(L.tsg_inject_alloc_failure(2, k))
    L.tsg_inject_alloc_failure(2, 0)


@pytest.fixture()
def make(built_lib):
    from tilespgemm_gb300 import Context
    made = []

    def m(**opts):
        made.append(Context(0, **opts))
        return made[-1]
    yield m
    for c in made:
        c.close()


def _lib():
    from tilespgemm_gb300 import _abi
    return _abi.lib()


def _scratch(c):
    return _lib().tsg_scratch_bytes(c.handle)


def _exact(C, A, B):
    rp, col, val = O.spgemm(A, B)
    assert np.array_equal(np.asarray(C.rowptr, np.int64), rp)
    assert np.array_equal(C.col, col) and np.array_equal(C.val, val)


BIG = dict(m=900, n=900, lens=[60, 9, 33], seed=91)


def _grown(c):
    """A context that keeps scratch: a call asks for it, the next one has it."""
    A = _rows(**BIG)
    for _ in range(2):
        _exact(c.spgemm(A, op="AA"), A, A)
    assert _scratch(c) > 0


def _calls():
    from tilespgemm_gb300 import matrices as M
    X = _rows(300, 300, [20, 5], 92)
    S = M.laplacian_2d(24)

    def plan(c):
        p = c.plan(X, op="AA")
        _exact(p.execute(np.asarray(X.val)), X, X)
        p.close()

    def batched_plan(c):
        p = c.plan_batched([X, X], op="AA")
        p.close()

    def tiles(c):
        assert c.spgemm_tiles(X, op="AA").numblk > 0

    return {"plan": plan, "batched_plan": batched_plan, "tiles": tiles,
            "small": lambda c: _exact(c.spgemm(S, op="AA"), S, S),
            "round_trip": lambda c: c.tiles_roundtrip(X)}


@pytest.mark.parametrize("name", sorted(_calls()))
@pytest.mark.parametrize("other", [False, True])
def test_idle_scratch_goes_to_a_call_that_needs_it(make, full, name, other):
    """`other`: the scratch is another context's."""
    c, keeper = make(), make()
    if not other:
        keeper = c
    _grown(keeper)
    full(1)
    _calls()[name](c)
    assert _lib().tsg_alloc_failure_pending(2) == 0
    assert _scratch(keeper) == 0
    A = _rows(**BIG)
    _exact(keeper.spgemm(A, op="AA"), A, A)


@pytest.mark.parametrize("name,small_path", [("heavy_items", 1), ("many_blocks", 1), ("stencil", 0), ("rmat9", 0)])
@pytest.mark.parametrize("out", ["host", "device"])
def test_products_without_room_run_without_what_is_kept(make, full, name, small_path, out):
    """Whichever allocation finds the memory full, the product is exact, and
    by tiles when it had to start again."""
    from test_rows_gpu import _b
    A, B, op = _cases()[name]
    ref = O.spgemm(A, _b(A, B, op))
    for k in range(1, 100):
        c = make(small_path=small_path)
        for _ in range(2):
            c.spgemm(A, B, op=op)
        kept, rows = _scratch(c), _lib().tsg_row_path_count()
        full(k)
        oc, _ = c.spgemm_raw(A, B, op=op, out=out)
        left = _lib().tsg_alloc_failure_pending(2)
        full(0)
        C = oc.download()
        oc.free()
        assert np.array_equal(np.asarray(C.rowptr, np.int64), ref[0])
        assert np.array_equal(C.col, ref[1]) and np.array_equal(C.val, ref[2])
        if left > 0:
            assert k > 1 and kept > 0
            return
        assert _scratch(c) == 0
        assert _lib().tsg_row_path_count() - rows <= small_path
        c.close()
    raise AssertionError("more allocations than expected")


def test_scratch_grows_again_later(make, full):
    """After a product had to be run again, the next calls do without scratch
    for a while, then keep it again."""
    c = make()
    A = _rows(**BIG)
    _grown(c)
    for rest in (1, 3):
        full(1)          # C's row pointer, columns or values: scratch has its own
        _exact(c.spgemm(A, op="AA"), A, A)
        assert _scratch(c) == 0
        for _ in range(rest):
            c.spgemm(A, op="AA")
            assert _scratch(c) == 0
        for _ in range(2):
            c.spgemm(A, op="AA")
        assert _scratch(c) > 0


@pytest.mark.parametrize("small_path", [0, 1])
def test_batches_without_room_run_without_what_is_kept(make, full, small_path):
    As = [_rows(m, m, [min(m, 20), 3], 93 + m) for m in (90, 1040, 37)]
    refs = [O.spgemm(A, A) for A in As]
    for k in range(1, 100):
        c = make(small_path=small_path)
        for _ in range(2):
            c.spgemm_batched(As, op="AA")
        full(k)
        got = c.spgemm_batched(As, op="AA")
        left = _lib().tsg_alloc_failure_pending(2)
        full(0)
        for C, ref in zip(got, refs):
            assert np.array_equal(np.asarray(C.rowptr, np.int64), ref[0])
            assert np.array_equal(C.col, ref[1]) and np.array_equal(C.val, ref[2])
        if left > 0:
            assert k > 1
            return
        c.close()
    raise AssertionError("more allocations than expected")


def test_scratch_is_given_back_beside_running_calls(make, full):
    """One thread's products keep and use scratch while another thread's calls
    take it back: every result is exact.  Both may meet a failure that the other
    armed, which is the documented error."""
    from tilespgemm_gb300 import TSGError, _abi
    A, X = _rows(**BIG), _rows(300, 300, [20, 5], 92)
    refA, refX = O.spgemm(A, A), O.spgemm(X, X)
    bad, stop = [], threading.Event()

    def same(C, ref):
        return (np.array_equal(np.asarray(C.rowptr, np.int64), ref[0]) and np.array_equal(C.col, ref[1])
                and np.array_equal(C.val, ref[2]))

    def products(c):
        while not stop.is_set():
            try:
                if not same(c.spgemm(A, op="AA"), refA):
                    bad.append("product")
            except TSGError as e:
                if e.status != _abi.ERR_OOM:
                    bad.append(str(e))

    ths = [threading.Thread(target=products, args=(make(),)) for _ in range(2)]
    taker = make()
    for t in ths:
        t.start()
    try:
        for i in range(150):
            full(1 + i % 3)
            try:
                p = taker.plan(X, op="AA")
                ok = same(p.execute(np.asarray(X.val)), refX)
                p.close()
                if not ok:
                    bad.append("plan")
            except TSGError as e:
                if e.status != _abi.ERR_OOM:
                    bad.append(str(e))
    finally:
        stop.set()
        for t in ths:
            t.join()
    assert not bad, bad[:3]
