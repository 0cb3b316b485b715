"""The waits of the solves whose blocks exchange values (exchange.cuh): each is
bounded, and one that runs out ends the call with MGPU_E_TIMEOUT (-5) and leaves
the case or the next call usable. The limit of one failed poll (tuning keys
exchange_spin_limit for the values, spin_limit for the sums' barrier) makes any
wait run out that does not find its value at the first poll; nothing hangs."""
import numpy as np
import pytest

from mixsolver_b200 import abi, cases
from mixsolver_b200 import solver as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib(gpu_lib):
    return gpu_lib


@pytest.fixture(autouse=True)
def _defaults():
    yield
    for key in ("exchange_spin_limit", "spin_limit", "resident_sms"):
        S.set_tuning(key, 0)


# FP64: 2 blocks sweep, the second waits for the first's values before its first
# level; mixed: 14 blocks exchange values after every polynomial step
@pytest.mark.parametrize("prec", [abi.PREC_FP64, abi.PREC_MIXED])
def test_value_wait_runs_out_then_case_recovers(prec):
    mesh, ctrl = cases.channel3d(24, 12, 12, seed=3, outer_max=3, order_fn=S.rcm_order)
    ctrl.precision, ctrl.lin_max = prec, 2000
    want = S.UnsCase(mesh, ctrl)
    ier, log = want.simple_run()
    assert ier == 0
    case = S.UnsCase(mesh, ctrl)
    S.set_tuning("exchange_spin_limit", 1)
    with pytest.raises(RuntimeError, match=r"status -5"):
        case.simple_run()
    S.set_tuning("exchange_spin_limit", 0)
    case.upload(u=np.zeros((mesh.ncells, 3)), p=np.zeros(mesh.ncells), flux=np.zeros(mesh.nfaces))
    ier, log2 = case.simple_run()
    assert ier == 0 and [r["lin_it"] for r in log] == [r["lin_it"] for r in log2]
    a, b = case.fields(), want.fields()
    for k in ("u", "p", "flux"):
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)


def _grid(nx, ny):
    """A 5-point system (1-based CSR) and a right-hand side."""
    n = nx * ny
    c = np.arange(n).reshape(ny, nx)
    lo = np.concatenate([c[:, :-1].ravel(), c[:-1].ravel()])
    hi = np.concatenate([c[:, 1:].ravel(), c[1:].ravel()])
    diag = np.bincount(lo, minlength=n) + np.bincount(hi, minlength=n) + 0.01
    rows, cols = np.concatenate([lo, hi, np.arange(n)]), np.concatenate([hi, lo, np.arange(n)])
    order = np.lexsort((cols, rows))
    ptr = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(rows, minlength=n), out=ptr[1:])
    vals = np.concatenate([np.full(2 * lo.size, -1.0), diag])[order]
    return (ptr + 1).astype(np.int32), (cols[order] + 1).astype(np.int32), vals, np.cos(np.arange(n) * 0.1)


# "spin_limit": the first wait of a solve in turns is the barrier of a sum
@pytest.mark.parametrize("key", ["exchange_spin_limit", "spin_limit"])
def test_wait_of_a_solve_in_turns_runs_out(key):
    ptr, col, val, b = _grid(150, 380)
    S.set_tuning("resident_sms", 12)
    solve = lambda: S.pcg_poly(ptr, col, val, b, np.zeros_like(b), 1e-9, 300)
    want = solve()
    S.set_tuning(key, 1)
    with pytest.raises(RuntimeError, match=r"status -5"):
        solve()
    S.set_tuning(key, 0)
    got = solve()
    assert got[1:] == want[1:] and want[3] == 0
    np.testing.assert_array_equal(got[0], want[0])
