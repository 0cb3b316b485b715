"""The shared-memory resident mixed solves (krylov_resident.cu) against the lanes
of a batch, which stream the same systems from memory: the same bits, for every
division of the rows that can go wrong (fewer rows than a super-chunk, one over,
ragged last blocks, several rows a thread, rows of 4 to 7 entries, orderings
whose halo is a few words or most of the system)."""
import numpy as np
import pytest

from mixsolver_b200 import abi, cases, meshgen
from mixsolver_b200 import solver as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib(gpu_lib):
    return gpu_lib


def _hex(nx, ny, nz, order):
    mesh = meshgen.box_hex(nx, ny, nz, jitter=0.05, seed=nx, zones=(5,) * 6)
    if order != "natural":
        mesh = meshgen.shuffle_cells(mesh, 3)
    if order == "rcm":
        return cases.rcm_renumber(mesh, S.rcm_order)
    return meshgen.sort_faces(mesh)


MESHES = {
    "64": lambda: _hex(4, 4, 4, "natural"),
    "255": lambda: _hex(17, 5, 3, "rcm"),
    "256": lambda: _hex(16, 4, 4, "rcm"),
    "257": lambda: _hex(257, 1, 1, "natural"),
    "513": lambda: _hex(57, 3, 3, "shuffled"),
    "2d": lambda: meshgen.cavity2d(37),
    "tet": lambda: meshgen.box_tet(9, wall_zone=5),
    "tet rcm": lambda: cases.rcm_renumber(meshgen.box_tet(19, wall_zone=5), S.rcm_order),
    "37k shuffled": lambda: _hex(41, 31, 29, "shuffled"),
    "39k rows over 148 blocks": lambda: _hex(39, 33, 30, "natural"),
    "several rows a thread": lambda: _hex(83, 47, 43, "rcm"),
}


@pytest.mark.parametrize("name", list(MESHES))
def test_resident_solves_bit_exact(name):
    mesh = MESHES[name]()
    ctrl = abi.Ctrl(rho=1.0, mu=1e-2, outer_max=2, outer_tol=0.0, lin_tol=1e-8, lin_max=500,
                    mom_solver=abi.MOM_JACOBI, precision=abi.PREC_MIXED,
                    bcs=[abi.BcSpec(zone=5, btype=abi.BC_WALL, lid=(2, 1.0, (1.0, 0.0, 0.0)))])
    if 4 in mesh.zone:
        ctrl.bcs.append(abi.BcSpec(zone=4, btype=abi.BC_SYMMETRY))
    one, lane = S.UnsCase(mesh, ctrl), S.UnsCase(mesh, ctrl)
    u = np.random.default_rng(1).standard_normal((mesh.ncells, 3)) * 0.1
    for c in (one, lane):
        c.upload(u=u)
    ier, log = one.simple_run(2)
    nrec, ier_b = S.CaseBatch([lane], policy=(32768, 1)).run(0, 2)
    assert ier == ier_b[0] == 0 and len(log) == nrec[0] == 2
    a, b = one.fields(), lane.fields()
    for k in a:
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)
