"""A numeric kernel that finds an entry outside the symbolic pass's structure
sets a device flag and leaves that part of C unwritten: every call that runs a
numeric step reports it and returns no result.  The flag is set behind the
kernels (tsg_inject_check_failure); nothing faults."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture()
def armed(built_lib):
    from tilespgemm_gb300 import Context, _abi
    L = _abi.lib()
    made = []

    def make(**opts):
        made.append(Context(0, **opts))
        return made[-1], lambda: _abi.check(L.tsg_inject_check_failure(1))
    yield make
    L.tsg_inject_check_failure(0)
    for c in made:
        c.close()


def _fails(call):
    from tilespgemm_gb300 import TSGError, _abi
    with pytest.raises(TSGError) as e:
        call()
    assert e.value.status == _abi.ERR_CUDA and "internal bound check" in str(e.value)


def _exact(C, A, B):
    rp, col, val = O.spgemm(A, B)
    assert np.array_equal(np.asarray(C.rowptr, np.int64), rp)
    assert np.array_equal(C.col, col) and np.array_equal(C.val, val)


@pytest.mark.parametrize("small_path", [0, 1])
@pytest.mark.parametrize("out", ["host", "device"])
@pytest.mark.parametrize("dense", [False, True])
def test_spgemm_reports_a_failed_check(armed, small_path, out, dense):
    """By tiles and by rows; `dense`: C's columns leave ahead of the values (host output by tiles)."""
    from tilespgemm_gb300 import matrices as M
    c, arm = armed(small_path=small_path)
    A = M.stencil_27(12, seed=2) if dense else M.random_sparse(500, 500, 20, seed=5)
    arm()
    _fails(lambda: c.spgemm_raw(A, op="AA", out=out))
    oc, _ = c.spgemm_raw(A, op="AA", out=out)      # the flag does not outlive its call
    _exact(oc.download(), A, A)
    oc.free()


def test_plans_tiles_and_batches_report_a_failed_check(armed):
    from tilespgemm_gb300 import matrices as M
    A = M.random_sparse(300, 300, 20, seed=6)
    for small_path in (0, 1):
        c, arm = armed(small_path=small_path)
        arm()
        _fails(lambda: c.spgemm_batched([A, A], op="AA"))
        for C in c.spgemm_batched([A, A], op="AA"):
            _exact(C, A, A)
        arm()
        _fails(lambda: c.spgemm_tiles(A, op="AA"))
        p = c.plan(A, op="AA")
        for out in ("host", "device"):
            arm()
            _fails(lambda: p.execute_raw(np.asarray(A.val), out=out))
        _exact(p.execute(np.asarray(A.val)), A, A)
        p.close()


def test_small_path_ignores_an_earlier_calls_flags(armed):
    """A repeated small product with host output runs one kernel with flags of
    its own: what another call left in the context's flags is not its error."""
    from tilespgemm_gb300 import matrices as M
    c, arm = armed()
    A, B = M.laplacian_2d(20), M.random_sparse(300, 300, 20, seed=7)
    for _ in range(2):
        _exact(c.spgemm(A, op="AA"), A, A)
    arm()
    _fails(lambda: c.spgemm(B, op="AA"))
    _exact(c.spgemm(A, op="AA"), A, A)
