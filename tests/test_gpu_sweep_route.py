"""Which FP64 factored solves run in shared memory (plan_sweep in
krylov_sweep.cu): by the names of the kernels that run, for systems on either
side of the rule's lines; those that krylov.cu solves give its bits."""
import numpy as np
import pytest
import torch
from torch.profiler import ProfilerActivity, profile

from mixsolver_b200 import meshgen
from mixsolver_b200 import solver as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib(gpu_lib):
    return gpu_lib


def _box(nx, ny, nz):
    n = nx * ny * nz
    c = np.arange(n).reshape(nz, ny, nx)
    lo = np.concatenate([c[:, :, :-1].ravel(), c[:, :-1].ravel(), c[:-1].ravel()])
    hi = np.concatenate([c[:, :, 1:].ravel(), c[:, 1:].ravel(), c[1:].ravel()])
    return n, lo, hi


def _tets(k):
    mesh = meshgen.box_tet(k, wall_zone=5)
    i = mesh.c1 > 0
    return mesh.ncells, mesh.c0[i].astype(np.int64) - 1, mesh.c1[i].astype(np.int64) - 1


# (graph, in shared memory): few blocks; more polls than 128 threads get through, but levels
# of at most 60 rows a block leave 448 of them; wide levels and 40 blocks that poll 3,453 rows each
ROUTES = {
    "4k box": (lambda: _box(16, 16, 16), True),
    "151k box": (lambda: _box(60, 60, 42), True),
    "83k tetrahedra": (lambda: _tets(24), False),
}


@pytest.mark.parametrize("name", list(ROUTES))
@pytest.mark.parametrize("method", ["cg_ic0", "bicgstab_ilu0"])
def test_route_of_factored_solves(name, method):
    graph, shared = ROUTES[name]
    n, lo, hi = graph()
    diag = np.bincount(lo, minlength=n) + np.bincount(hi, minlength=n) + 0.1
    rows, cols = np.concatenate([lo, hi, np.arange(n)]), np.concatenate([hi, lo, np.arange(n)])
    order = np.lexsort((cols, rows))
    ptr = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(rows, minlength=n), out=ptr[1:])
    args = ((ptr + 1).astype(np.int32), (cols[order] + 1).astype(np.int32),
            np.concatenate([np.full(2 * lo.size, -1.0), diag])[order], np.cos(0.1 * np.arange(n)), np.zeros(n))
    solve = getattr(S, method)
    torch.zeros(1).cuda()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        x, it, res, ierr = solve(*args, 1e-9, 300)
        torch.cuda.synchronize()
    names = [e.name for e in prof.events() if "k_pcg" in e.name or "k_bicgstab" in e.name]
    assert ierr == 0 and res <= 1e-9
    assert names and all(("sweep" in k) == shared for k in names), names
