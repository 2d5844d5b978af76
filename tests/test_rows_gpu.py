"""The row path of tsg_spgemm (tsg_rows.cu): products whose tiles are nearly
empty, or small ones, run row by row.  C must equal the oracle's and the
tiled pipeline's bit for bit: both accumulate each entry as fma over A's row
order, then B's.  The sizes sit at the path's edges: its blocks of 1,024
columns, the threads of a step, rows of one item and of many, dense blocks,
rows wider than one bitmap window."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rctx(built_lib):
    from tilespgemm_gb300 import Context
    c = Context(0)
    yield c
    c.close()


def _rows(m, n, lens, seed):
    """m rows of the given lengths, distinct ascending random columns."""
    from tilespgemm_gb300.api import CSR
    rng = np.random.default_rng(seed)
    lens = np.minimum(np.resize(np.asarray(lens, np.int64), m), n)
    rp = np.zeros(m + 1, np.int64)
    np.cumsum(lens, out=rp[1:])
    col = np.concatenate([np.sort(rng.choice(n, int(c), replace=False)) for c in lens] or [np.empty(0)])
    return CSR(m, n, rp, col.astype(np.int32), rng.uniform(-1.0, 1.0, int(rp[-1])))


def _spread(X, f):
    """X's columns f apart."""
    from tilespgemm_gb300.api import CSR
    return CSR(X.m, X.n * f, X.rowptr, X.col * np.int32(f), X.val)


def _cases():
    from tilespgemm_gb300 import matrices as M
    return {
        "one_block": (_rows(150, 150, [5, 40, 0, 149], 1), None, "AA"),
        "n1023": (_rows(200, 1023, [30], 2), _rows(1023, 1023, [17, 33, 0, 128], 3), "AB"),
        "n1024": (_rows(200, 300, [30], 4), _rows(300, 1024, [31, 32, 129], 5), "AB"),
        "n1025": (_rows(200, 300, [30], 6), _rows(300, 1025, [1, 64, 127], 7), "AB"),
        "one_entry_shares": (_rows(130, 4000, [700, 64, 33], 8), _rows(4000, 9001, [1, 0, 2], 9), "AB"),
        "many_blocks": (_rows(90, 500, [40, 3], 10), _rows(500, 70001, [300, 7, 1200], 11), "AB"),
        "two_windows": (_rows(60, 400, [12, 90], 12), _rows(400, 300007, [20, 900], 13), "AB"),
        "heavy_items": (_rows(7, 600, [500, 300, 20], 14), _rows(600, 40013, [700, 40, 2500], 15), "AB"),
        "heavy_windows": (_rows(5, 400, [380, 40], 16), _rows(400, 290003, [3000, 0, 9000], 17), "AB"),
        "dense_blocks": (_rows(40, 200, [150, 60], 18), _rows(200, 5000, [2500, 4000, 8], 19), "AB"),
        "full_rows": (_rows(6, 90, [90], 20), _rows(90, 2049, [2049], 21), "AB"),
        "sort_classes": (_rows(700, 60, [1], 22),
                         _rows(60, 120007, [1, 31, 33, 127, 128, 129, 255, 256, 257, 511, 512, 513, 0], 23), "AB"),
        "sort_batches": (_rows(150, 300, [64, 33, 32, 65, 130, 7], 24), _rows(300, 100003, [0, 4, 8, 3, 1], 25), "AB"),
        "sort_repeats": (_rows(200, 50, [4, 3, 1, 5], 26), _spread(_rows(50, 150, [128, 40, 100], 27), 900), "AB"),
        "wide_a": (_rows(20, 9000, [5000, 2049, 2048, 10, 0, 8999], 28), _rows(9000, 3000, [3, 0, 1], 29), "AB"),
        "rmat9": (M.rmat(9, 8, seed=3), None, "AAT"),
        "rmat12": (M.rmat(12, 8, seed=4), None, "AA"),
        "stencil": (M.stencil_27(11, seed=2), None, "AAT"),
        "empty_rows": (M.random_sparse(3000, 3000, 40, seed=16, empty_rows=0.5), None, "AA"),
        "unsorted_b": (M.random_sparse(600, 600, 30, seed=17, unsorted=True), None, "AA"),
        "repeated_b": (M.random_sparse(600, 600, 30, seed=18, dup=True), None, "AA"),
    }


def _b(A, B, op):
    from tilespgemm_gb300.api import CSR
    if op == "AB":
        return B
    if op == "AA":
        return A
    tp, tr, tv = O.transpose(A)
    return CSR(A.n, A.m, tp, tr, tv)


def _check(C, ref):
    assert np.array_equal(np.asarray(C.rowptr, np.int64), ref[0])
    assert np.array_equal(C.col, ref[1])
    assert np.array_equal(C.val, ref[2])


@pytest.mark.parametrize("name", sorted(_cases()))
def test_rows_match_oracle_and_tiles(rctx, ctx, name):
    A, B, op = _cases()[name]
    ref = O.spgemm(A, _b(A, B, op))
    _check(rctx.spgemm(A, B, op=op), ref)
    _check(ctx.spgemm(A, B, op=op), ref)       # the tiled pipeline


def test_rows_many_products_match_tiles(rctx, ctx):
    """Over 400 M products: rows of up to 2,048 entries are light, not 4,096."""
    A = _rows(13000, 8000, [6, 7, 12, 15, 16, 230, 230, 230], 30)
    B = _rows(8000, 8200, [360], 31)
    C, D = rctx.spgemm(A, B, op="AB"), ctx.spgemm(A, B, op="AB")
    _check(C, (np.asarray(D.rowptr, np.int64), D.col, D.val))


@pytest.mark.parametrize("bits", [32, 64])
def test_rows_device_operands_and_output(rctx, bits):
    import torch
    A, B, op = _cases()["many_blocks"]
    ref = O.spgemm(A, B)
    dA, dB = A.to_device(0), B.to_device(0)
    for X in (dA, dB):
        X.rowptr = X.rowptr.to(torch.int64 if bits == 64 else torch.int32)
    oc, _ = rctx.spgemm_raw(dA, dB, op=op, out="device")
    assert oc.where == "device"
    _check(oc.download(), ref)
    oc.free()


def test_rows_allocation_failures(rctx):
    """Every device and pinned allocation of a call failing in turn: an error,
    and the next call is exact."""
    from tilespgemm_gb300 import _abi
    lib = _abi.lib()
    A, B, op = _cases()["heavy_items"]
    ref = O.spgemm(A, B)
    for kind in (0, 1):
        for k in range(1, 100):
            _abi.check(lib.tsg_inject_alloc_failure(kind, k))
            try:
                C = rctx.spgemm(A, B, op=op)
                assert lib.tsg_alloc_failure_pending(kind) > 0
                _abi.check(lib.tsg_inject_alloc_failure(kind, 0))
                _check(C, ref)
                break
            except _abi.TSGError as e:
                assert "TSG_ERR_OOM" in str(e)
                assert lib.tsg_alloc_failure_pending(kind) == 0
            _check(rctx.spgemm(A, B, op=op), ref)
        else:
            raise AssertionError("more allocations than expected")


def test_rows_bad_columns(rctx):
    from tilespgemm_gb300 import _abi
    from tilespgemm_gb300.api import CSR
    A, B, op = _cases()["n1024"]
    col = B.col.copy()
    col[5] = B.n
    with pytest.raises(_abi.TSGError):
        rctx.spgemm(A, CSR(B.m, B.n, B.rowptr, col, B.val), op=op)
    _check(rctx.spgemm(A, B, op=op), O.spgemm(A, B))


@pytest.mark.parametrize("op", ["AA", "AAT", "AB"])
def test_batched_rows(rctx, op):
    """A batch by the row path (instances that start inside a block, widths
    around one, a heavy row with several items): each equals its oracle."""
    shapes = [(90, 90), (1040, 1040), (1, 1), (2100, 2100), (37, 37), (5000, 5000)]
    if op != "AA":
        shapes = [(m, n + 3 * i) for i, (m, n) in enumerate(shapes)]
    As = [_rows(m, n, [min(n, 20), 3, min(n, 90)], 40 + i) for i, (m, n) in enumerate(shapes)]
    As.append(_rows(12, 12 if op == "AA" else 300, [250, 5], 50))
    Bs = None
    if op == "AB":
        Bs = [_rows(A.n, 700 + 2000 * i, [40, 0, 600], 60 + i) for i, A in enumerate(As)]
    got = rctx.spgemm_batched(As, Bs, op=op)
    for i, A in enumerate(As):
        _check(got[i], O.spgemm(A, _b(A, Bs[i] if Bs else None, op)))
