"""The quotient of the shared-memory sweeps (krylov_sweep.cu), which takes the
place of a division where no intermediate can over- or underflow, against
krylov.cu's division, bit for bit: diagonal systems, whose first iteration
divides each right-hand side by its diagonal (ILU(0)) or twice by its root
(IC(0)). Rows next to the exponents where the quotient hands over to the
division, zeros, subnormal operands and results, mantissas of all ones and
next to a power of two. A dense 8 x 8 block with a zero right-hand side sends
a system to krylov.cu (more than 6 entries on one side of a diagonal)."""
import numpy as np
import pytest

from mixsolver_b200 import solver as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib(gpu_lib):
    return gpu_lib


def _operands():
    """(dividends, divisors): r^2, r / d and r^2 / d stay finite, so that the sums do."""
    rng = np.random.default_rng(11)
    one = 2.0 ** -52
    mant = np.array([1.0, 1.0 + one, 1.0 + 2 * one, 1.5, 2.0 - one, 2.0 - 2 * one])
    r, d = [], []
    for er in (-1074, -1060, -1022, -700, -512, -511, -510, -300, 0, 200, 400):
        for ed in (-1030, -900, -300, -225, -224, -223, -222, -50, 0, 50, 222, 223, 224, 225, 226, 300, 900, 1000):
            if 2 * er - ed > 900 or er - ed > 900:
                continue
            k = 12
            a = np.concatenate([mant, rng.uniform(1.0, 2.0, k)])
            b = np.concatenate([rng.permutation(mant), rng.uniform(1.0, 2.0, k)])
            r.append(np.ldexp(a, er) * rng.choice([-1.0, 1.0], a.size))
            d.append(np.ldexp(b, ed))
    r.append(np.array([0.0, -0.0, 0.0]))
    d.append(np.array([3.0, 5.0, np.ldexp(1.0, -1030)]))
    r, d = np.concatenate(r), np.concatenate(d)
    # the bulk: ordinary operands, every one a chance for a wrong last bit
    n = 20000
    r = np.concatenate([r, rng.standard_normal(n) * 2.0 ** rng.integers(-200, 200, n)])
    d = np.concatenate([d, rng.uniform(1.0, 2.0, n) * 2.0 ** rng.integers(-200, 200, n)])
    return r, d


@pytest.mark.parametrize("method", ["cg_ilu0", "cg_ic0"])
def test_quotients_are_the_divisions(method):
    r, d = _operands()
    n, tail = r.size, 8
    solve = getattr(S, method)
    ptr = np.arange(1, n + 2, dtype=np.int32)
    col = np.arange(1, n + 1, dtype=np.int32)
    x, it, res, ierr = solve(ptr, col, d, r, np.zeros(n), 1e-30, 1)
    block = np.where(np.eye(tail, dtype=bool), 9.0, -1.0).ravel()
    ptr2 = np.concatenate([ptr, n + 1 + tail * np.arange(1, tail + 1)]).astype(np.int32)
    col2 = np.concatenate([col, np.tile(np.arange(n + 1, n + tail + 1), tail)]).astype(np.int32)
    y, it2, res2, ierr2 = solve(ptr2, col2, np.concatenate([d, block]), np.concatenate([r, np.zeros(tail)]),
                                np.zeros(n + tail), 1e-30, 1)
    assert np.isfinite(x).all() and np.count_nonzero(x) > 0.9 * n
    assert (it, res, ierr) == (it2, res2, ierr2)
    np.testing.assert_array_equal(x.view(np.int64), y[:n].view(np.int64))
