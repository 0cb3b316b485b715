"""The ILU(0) / IC(0) solves on rows in shared memory (krylov_sweep.cu) against
krylov.cu's, bit for bit. A system goes to krylov.cu when a row has more than 6
entries on one side of the diagonal, so each system is solved as it is and with
a decoupled dense 8 x 8 block after it (zero right-hand side: its rows add zeros
to every sum). Sizes: one row short of and past a block's lists, several blocks,
levels narrower and wider than the sweeping warps, 2 to 6 entries a side."""
import numpy as np
import pytest

from mixsolver_b200 import cases, meshgen
from mixsolver_b200 import solver as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib(gpu_lib):
    return gpu_lib


def _hex(nx, ny, nz, order):
    mesh = meshgen.box_hex(nx, ny, nz, zones=(5,) * 6)
    if order == "natural":
        return mesh
    mesh = meshgen.shuffle_cells(mesh, 3)
    return cases.rcm_renumber(mesh, S.rcm_order) if order == "rcm" else mesh


MESHES = {
    "9": lambda: meshgen.cavity2d(3),
    "2d 33": lambda: meshgen.cavity2d(33),
    "2d 70": lambda: meshgen.cavity2d(70),
    "hex 13": lambda: _hex(13, 13, 13, "natural"),
    "hex rcm": lambda: _hex(31, 19, 17, "rcm"),
    "hex shuffled": lambda: _hex(11, 9, 8, "shuffled"),
    "hex 36k": lambda: _hex(41, 31, 28, "natural"),
    "hex 36k rcm": lambda: _hex(41, 31, 28, "rcm"),
    "tet": lambda: meshgen.box_tet(11, wall_zone=5),
    "tet rcm": lambda: cases.rcm_renumber(meshgen.box_tet(14, wall_zone=5), S.rcm_order),
}


def _system(mesh, symmetric, tail):
    """1-based CSR of the mesh's graph with seeded coefficients, `tail` more rows dense."""
    rng = np.random.default_rng(7)
    i = mesh.c1 > 0
    a, b = mesh.c0[i].astype(np.int64) - 1, mesh.c1[i].astype(np.int64) - 1
    w = np.exp(rng.uniform(-1.0, 1.0, a.size))
    v = w if symmetric else w * rng.uniform(0.7, 1.0, a.size)
    n = mesh.ncells
    diag = np.bincount(a, w, n) + np.bincount(b, w, n) + 0.01
    t = np.arange(tail) + n
    tr, tc = (m.ravel() for m in np.meshgrid(t, t, indexing="ij"))
    rows = np.concatenate([a, b, np.arange(n), tr])
    cols = np.concatenate([b, a, np.arange(n), tc])
    vals = np.concatenate([-w, -v, diag, np.where(tr == tc, 9.0, -1.0)])
    order = np.lexsort((cols, rows))
    ptr = np.zeros(n + tail + 1, np.int64)
    np.cumsum(np.bincount(rows, minlength=n + tail), out=ptr[1:])
    rhs = np.concatenate([rng.standard_normal(n), np.zeros(tail)])
    return (ptr + 1).astype(np.int32), (cols[order] + 1).astype(np.int32), vals[order], rhs


@pytest.mark.parametrize("name", list(MESHES))
@pytest.mark.parametrize("method", ["cg_ic0", "cg_ilu0", "bicgstab_ilu0"])
def test_sweep_solves_bit_exact(name, method):
    mesh = MESHES[name]()
    n = mesh.ncells
    solve = getattr(S, method)
    ptr, col, val, b = _system(mesh, method != "bicgstab_ilu0", 0)
    x, it, res, ierr = solve(ptr, col, val, b, np.zeros(n), 1e-9, 300)
    ptr, col, val, b = _system(mesh, method != "bicgstab_ilu0", 8)
    y, it2, res2, ierr2 = solve(ptr, col, val, b, np.zeros(n + 8), 1e-9, 300)
    assert ierr == ierr2 == 0 and it == it2 and res == res2
    np.testing.assert_array_equal(x, y[:n])
