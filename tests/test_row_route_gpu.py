"""Which products run row by row: the row path and the tiles give the same
bits, so tsg_row_path_count tells which one made them."""
import numpy as np
import pytest

from oracle import oracle as O
from test_rows_gpu import _b, _cases, _rows, rctx  # noqa: F401  (rctx: the fixture)

pytestmark = pytest.mark.gpu


def _count():
    from tilespgemm_gb300 import _abi
    return _abi.lib().tsg_row_path_count()


def _went(call):
    """The call's result and the products it ran by rows."""
    before = _count()
    out = call()
    return out, _count() - before


def _check(C, ref):
    assert np.array_equal(np.asarray(C.rowptr, np.int64), ref[0])
    assert np.array_equal(C.col, ref[1])
    assert np.array_equal(C.val, ref[2], equal_nan=True)
    live = ~np.isnan(ref[2])
    assert np.array_equal(np.signbit(C.val[live]), np.signbit(ref[2][live]))


@pytest.mark.parametrize("name", sorted(_cases()))
def test_cases_take_the_row_path(rctx, ctx, name):  # noqa: F811
    A, B, op = _cases()[name]
    rows = name not in ("unsorted_b", "repeated_b")
    assert _went(lambda: rctx.spgemm(A, B, op=op))[1] == int(rows)
    assert _went(lambda: ctx.spgemm(A, B, op=op))[1] == 0          # small_path = 0


def test_many_products_take_the_row_path(rctx):  # noqa: F811
    A = _rows(13000, 8000, [6, 7, 12, 15, 16, 230, 230, 230], 30)
    B = _rows(8000, 8200, [360], 31)
    assert _went(lambda: rctx.spgemm_raw(A, B, op="AB", out="device"))[1] == 1


def _special(X, seed):
    """X with infinities, NaN, zeros of both signs and subnormals among its values."""
    from tilespgemm_gb300.api import CSR
    v = X.val.copy()
    rng = np.random.default_rng(seed)
    for x in (np.inf, -np.inf, np.nan, 0.0, -0.0, 5e-324, 1.7e308):
        v[rng.integers(0, v.size, max(1, v.size // 200))] = x
    return CSR(X.m, X.n, X.rowptr, X.col, v)


def _near(m, lens, lo, hi, n, seed):
    """m rows of n columns whose entries all lie in [lo, hi)."""
    from tilespgemm_gb300.api import CSR
    X = _rows(m, hi - lo, lens, seed)
    return CSR(m, n, X.rowptr, (X.col + lo).astype(np.int32), X.val)


def _more():
    from tilespgemm_gb300 import matrices as M
    return {
        # A in any order and with repeated columns: only B's rows have to increase
        "a_unsorted": (M.random_sparse(400, 300, 30, seed=61, unsorted=True, dup=True), _rows(300, 4000, [50, 7, 200], 62)),
        "special_items": (_special(_rows(90, 500, [40, 3], 63), 64), _special(_rows(500, 70001, [300, 7, 1200], 65), 66)),
        "special_sorted": (_special(_rows(150, 300, [64, 33, 7], 67), 68), _special(_rows(300, 100003, [4, 8, 3], 69), 70)),
        # too many columns for the sort's 32-bit keys
        "no_sort": (_rows(200, 300, [40, 12], 71), _near(300, [6, 11], 8200000, 8300000, 8400000, 72)),
    }


@pytest.mark.parametrize("name", sorted(_more()))
def test_more_forms_by_rows(rctx, name):  # noqa: F811
    A, B = _more()[name]
    C, went = _went(lambda: rctx.spgemm(A, B, op="AB"))
    assert went == 1
    _check(C, O.spgemm(A, B))


def test_too_wide_rows_go_by_tiles(rctx):  # noqa: F811
    """Rows over more than 4,096 blocks of columns, known only after the
    products were counted: the call starts again by tiles, alone and in a batch."""
    A, B = _rows(60, 50, [30, 4], 73), _rows(50, 5000000, [200, 33], 74)
    C, went = _went(lambda: rctx.spgemm(A, B, op="AB"))
    assert went == 0
    _check(C, O.spgemm(A, B))
    A2, B2 = _rows(90, 120, [30, 7], 75), _rows(120, 900, [80, 5], 76)
    got, went = _went(lambda: rctx.spgemm_batched([A2, A, A2], [B2, B, B2], op="AB"))
    assert went == 0
    for X, Y, Z in zip(got, (A2, A, A2), (B2, B, B2)):
        _check(X, O.spgemm(Y, Z))


@pytest.mark.parametrize("op", ["AA", "AAT", "AB"])
def test_batches_by_rows_on_the_device(rctx, op):  # noqa: F811
    As = [_rows(m, m, [min(m, 20), 3, min(m, 90)], 80 + m) for m in (90, 1040, 37, 2100)]
    Bs = [_rows(A.n, 700 + 500 * i, [40, 0, 300], 81 + i) for i, A in enumerate(As)] if op == "AB" else None
    dB = [B.to_device(0) for B in Bs] if Bs else None
    (outs, _), went = _went(lambda: rctx.spgemm_batched_raw([A.to_device(0) for A in As], dB, op=op, out="device"))
    assert went == 1
    for i, (A, oc) in enumerate(zip(As, outs)):
        _check(oc.download(), O.spgemm(A, _b(A, Bs[i] if Bs else None, op)))
        oc.free()


@pytest.fixture()
def free_memory():
    from tilespgemm_gb300 import _abi
    L = _abi.lib()
    yield lambda n: _abi.check(L.tsg_inject_free_memory(n))
    L.tsg_inject_free_memory(-1)


@pytest.mark.parametrize("name", ["one_block", "many_blocks", "heavy_windows", "rmat9", "sort_classes"])
def test_tables_without_room(rctx, free_memory, name):  # noqa: F811
    """With more and more free memory: first by tiles, then by rows with the
    bitmaps made again, then with them kept; always the same C."""
    A, B, op = _cases()[name]
    ref = O.spgemm(A, _b(A, B, op))
    ways = []
    for n in [0] + [1 << e for e in range(10, 44, 3)]:
        free_memory(n)
        C, went = _went(lambda: rctx.spgemm(A, B, op=op))
        _check(C, ref)
        ways.append(went)
    assert ways[0] == 0 and ways[-1] == 1 and ways == sorted(ways)


def test_items_of_light_rows_fit_their_bound(rctx):  # noqa: F811
    """Rows of few entries over more than 256 and 512 blocks: two and three
    items each, as many as their bound; also with rows past LIGHT_MANY among them."""
    for n in (300007, 600011):
        A, B = _rows(700, 400, [25, 30, 26, 90], 85), _rows(400, n, [22, 31, 25], 86)
        C, went = _went(lambda: rctx.spgemm(A, B, op="AB"))
        assert went == 1
        _check(C, O.spgemm(A, B))


def _spaced(m, n, lens, seed):
    """m rows of the given lengths over n columns: one random column of each of
    so many equal parts of them, so that hardly two share a tile."""
    from tilespgemm_gb300.api import CSR
    rng = np.random.default_rng(seed)
    lens = np.resize(np.asarray(lens, np.int64), m)
    rp = np.zeros(m + 1, np.int64)
    np.cumsum(lens, out=rp[1:])
    part = n // np.maximum(lens, 1)
    at = np.arange(rp[-1]) - np.repeat(rp[:-1], lens)
    wide = np.repeat(part, lens)
    col = at * wide + (rng.random(at.size) * wide).astype(np.int64)
    return CSR(m, n, rp, col.astype(np.int32), rng.uniform(-1.0, 1.0, int(rp[-1])))


def _band(n, h, seed):
    from tilespgemm_gb300.api import CSR
    c = np.arange(n)[:, None] + np.arange(-h, h + 1)[None, :]
    ok = (c >= 0) & (c < n)
    rp = np.zeros(n + 1, np.int64)
    np.cumsum(ok.sum(1), out=rp[1:])
    return CSR(n, n, rp, c[ok].astype(np.int32), np.random.default_rng(seed).uniform(-1.0, 1.0, int(rp[-1])))


@pytest.mark.parametrize("m,clustered,rows", [(65536, True, 1), (65537, True, 0), (65537, False, 1)])
def test_many_clustered_rows_go_by_tiles(rctx, ctx, m, clustered, rows):  # noqa: F811
    """Under 24 M products, on both sides of 65,536 rows: there the rows' fixed
    cost counts, and tiles that hold several entries a row are cheaper."""
    A = _band(m, 6, 95) if clustered else _spaced(m, m, [13], 96)
    op = "AA"
    C, went = _went(lambda: rctx.spgemm(A, op=op))
    assert went == rows
    D, none = _went(lambda: ctx.spgemm(A, op=op))
    assert none == 0
    _check(C, (np.asarray(D.rowptr, np.int64), D.col, D.val))
