"""The pressure solve that takes its pages in turns (k_pcg_paged in
krylov_resident.cu) against the streaming kernel, bit for bit, for every page
size the plan can choose, both row widths and the ends of its ranges: ragged
last pages, degrees below and not divisible by the steps of a turn, restarts
from the true residual, solves that run out of iterations. The tuning key
resident_sms lets systems of some 50,000 rows be larger than the SMs it counts
on. The same system goes to the streaming kernel with one more entry, of value
zero and without a transposed one: only symmetric patterns are divided."""
import numpy as np
import pytest
import torch
from torch.profiler import ProfilerActivity, profile

from mixsolver_b200 import solver as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib(gpu_lib):
    yield gpu_lib
    S.set_tuning("resident_sms", 0)


def _graph(nx, ny, nz, window):
    """Faces of a box whose cells are numbered x fastest, then mixed within windows."""
    n = nx * ny * nz
    new = np.arange(n)
    rng = np.random.default_rng(1)
    for s in range(0, n if window else 0, window or 1):
        e = min(n, s + window)
        new[s:e] = s + rng.permutation(e - s)
    c = new.reshape(nz, ny, nx)
    lo = np.concatenate([c[:, :, :-1].ravel(), c[:, :-1].ravel(), c[:-1].ravel()])
    hi = np.concatenate([c[:, :, 1:].ravel(), c[:, 1:].ravel(), c[1:].ravel()])
    return n, lo, hi


def _system(n, lo, hi):
    """1-based CSR with seeded coefficients, a right-hand side, and the CSR with the unpaired entry."""
    rng = np.random.default_rng(2)
    k = np.exp(rng.uniform(-1.5, 1.5, lo.size))
    diag = np.bincount(lo, k, n) + np.bincount(hi, k, n) + 1e-3
    rows = np.concatenate([lo, hi, np.arange(n)])
    cols = np.concatenate([hi, lo, np.arange(n)])
    vals = np.concatenate([-k, -k, diag])

    def csr(r, c, v):
        order = np.lexsort((c, r))
        ptr = np.zeros(n + 1, np.int64)
        np.cumsum(np.bincount(r, minlength=n), out=ptr[1:])
        return (ptr + 1).astype(np.int32), (c[order] + 1).astype(np.int32), v[order]

    width = np.bincount(rows, minlength=n)
    r = int(np.argmin(width))  # a corner: one entry more does not widen the widest row
    assert width[r] < width.max()
    c = next(c for c in range(n) if c != r and c not in cols[rows == r])
    return (csr(rows, cols, vals), csr(np.append(rows, r), np.append(cols, c), np.append(vals, 0.0)),
            rng.standard_normal(n))


# (box, window of the numbering, SMs counted on): super-chunks of a page that the plan takes
DIVISIONS = {
    "7 entries, 5": ((31, 29, 98), 2500, 24),
    "7 entries, 6": ((60, 50, 29), 1000, 24),
    "7 entries, 7": ((31, 29, 42), 0, 8),
    "5 entries, 5": ((300, 188, 1), 6000, 12),
    "5 entries, 6": ((300, 188, 1), 5000, 12),
    "5 entries, 7": ((300, 188, 1), 4000, 12),
    "5 entries, 8": ((300, 188, 1), 3000, 12),
    "5 entries, 9": ((300, 188, 1), 1000, 12),
    "5 entries, 9, short reach": ((37, 1524, 1), 0, 12),
}


@pytest.mark.parametrize("name", list(DIVISIONS))
def test_paged_solves_bit_exact(name):
    box, window, sms = DIVISIONS[name]
    paired, unpaired, b = _system(*_graph(*box, window))
    x0 = 0.1 * np.cos(np.arange(b.size))
    S.set_tuning("resident_sms", sms)
    # (tolerance, iterations, degree); 1e-15 is below what a restart reaches
    for tol, maxit, degree in ((1e-9, 400, 24), (1e-9, 4000, 2), (1e-8, 400, 64), (1e-10, 4, 9), (1e-15, 40, 24)):
        x, it, res, ierr = S.pcg_poly(*paired, b, x0, tol, maxit, cheb_degree=degree)
        y, it2, res2, ierr2 = S.pcg_poly(*unpaired, b, x0, tol, maxit, cheb_degree=degree)
        assert (it, res, ierr) == (it2, res2, ierr2), (tol, maxit, degree)
        assert ierr == (1 if tol < 1e-9 and maxit <= 40 else 0)
        np.testing.assert_array_equal(x, y, err_msg=str((tol, maxit, degree)))
    x, it, res, ierr = S.pcg_poly(*paired, np.zeros_like(b), x0, 1e-9, 10)
    assert (it, res, ierr) == (0, 0.0, 0) and not x.any()


def test_window_beyond_the_flags_is_streamed():
    """A reach of 196,200 rows makes 12,288 window words, 48 KB of flags in the
    kernel that counts the halo: not divided, and solved all the same."""
    n, reach = 196_400, 196_200
    lo = np.concatenate([np.arange(n - 1), [0]])
    hi = np.concatenate([np.arange(1, n), [reach]])
    paired, unpaired, b = _system(n, lo, hi)
    got, want = (S.pcg_poly(*m, b, np.zeros(n), 1e-9, 400) for m in (paired, unpaired))
    assert got[1:] == want[1:] and got[3] == 0
    np.testing.assert_array_equal(got[0], want[0])


# 524,288 rows mixed within 500: does not fit in shared memory, still hits L2 (in turns an
# iteration took 380 us instead of 214); 1.44M rows: beyond L2 (921 us instead of 1,033)
@pytest.mark.parametrize("box, window, kernel", [((128, 64, 64), 500, "k_pcg_mixed"),
                                                 ((113, 113, 113), 0, "k_pcg_paged")])
def test_turns_only_where_they_pay(box, window, kernel):
    S.set_tuning("resident_sms", 0)
    paired, _, b = _system(*_graph(*box, window))
    torch.zeros(1).cuda()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        S.pcg_poly(*paired, b, np.zeros_like(b), 1e-8, 3)
        torch.cuda.synchronize()
    names = [e.name for e in prof.events() if "k_pcg" in e.name]
    assert names and all(kernel in k for k in names), names
