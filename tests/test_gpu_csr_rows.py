"""Stand-alone solves of CSR rows whose columns do not ascend: a larger column
before the diagonal hides it (the diagonal counts as missing, as it did for the
search along the row); entries out of order behind the diagonal are solved."""
import numpy as np
import pytest

from mixsolver_b200 import solver as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib(gpu_lib):
    return gpu_lib


def _system(n=900, nx=30):
    """A 5-point system, its solution and right-hand side (1-based CSR)."""
    i = np.arange(n)
    e = i[i % nx != nx - 1]
    lo, hi = np.concatenate([e, i[:-nx]]), np.concatenate([e + 1, i[:-nx] + nx])
    rng = np.random.default_rng(5)
    k = rng.uniform(0.5, 2.0, lo.size)
    d = np.bincount(lo, k, n) + np.bincount(hi, k, n) + 0.1
    rows, cols = np.concatenate([lo, hi, i]), np.concatenate([hi, lo, i])
    order = np.lexsort((cols, rows))
    ptr = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(rows, minlength=n), out=ptr[1:])
    cols, vals = cols[order], np.concatenate([-k, -k, d])[order]
    x = rng.standard_normal(n)
    b = np.bincount(rows[order], vals * x[cols], n)
    return (ptr + 1).astype(np.int32), (cols + 1).astype(np.int32), vals, x, b


def _reorder(ptr, col, val, row, order):
    """The entries of a row in another order (positions within the row)."""
    col, val = col.copy(), val.copy()
    s = slice(ptr[row] - 1, ptr[row + 1] - 1)
    col[s], val[s] = col[s][order], val[s][order]
    return col, val


def test_larger_column_before_the_diagonal_hides_it():
    ptr, col, val, _, b = _system()
    col, val = _reorder(ptr, col, val, 455, [4, 0, 1, 2, 3])
    x0 = np.zeros_like(b)
    for solve, code in ((S.cg_ic0, 11), (S.cg_ilu0, 11), (S.bicgstab_ilu0, 11), (S.cg_jacobi, 2),
                        (S.bicgstab_jacobi, 12)):
        x, it, res, ierr = solve(ptr, col, val, b, x0, 1e-9, 200)
        assert (it, res, ierr) == (0, 0.0, code), solve.__name__
    with pytest.raises(RuntimeError, match="no diagonal"):
        S.pcg_poly(ptr, col, val, b, x0, 1e-9, 200)


@pytest.mark.parametrize("name", ["cg_jacobi", "bicgstab_jacobi", "cg_ilu0", "bicgstab_ilu0", "pcg_poly"])
def test_rows_out_of_order_behind_the_diagonal_are_solved(name):
    ptr, col, val, x, b = _system()
    for row in (40, 451, 700):
        col, val = _reorder(ptr, col, val, row, [0, 1, 2, 4, 3])
    y, it, res, ierr = getattr(S, name)(ptr, col, val, b, np.zeros_like(b), 1e-10, 500)
    assert ierr == 0 and res <= 1e-10
    # |x - y| <= |A^-1| |r|: the smallest eigenvalue is at least the reaction term, 0.1
    assert np.linalg.norm(x - y) <= 1e-9 * np.linalg.norm(b) * 1.1


def test_unpaired_entries_are_refused_by_ic0():
    ptr, col, val, _, b = _system()
    col, val = _reorder(ptr, col, val, 451, [0, 1, 2, 4, 3])
    with pytest.raises(RuntimeError, match="symmetric"):
        S.cg_ic0(ptr, col, val, b, np.zeros_like(b), 1e-9, 200)
