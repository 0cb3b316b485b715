"""The measured workloads: what a user of the library has it do, through its public
entry points, from the smallest cavity to three million tetrahedra.

A pass of a flow case is the coupling loop's call: the current fields go up from
page-locked host arrays, the case advances a few outer iterations or one time step,
and the new fields come back into page-locked arrays. A pass of a linear system is
one solver call on a host CSR system, as `mod_uns_linsolver` is called.
"""
import functools

import numpy as np
import torch

from mixsolver_b200 import abi, cases, meshgen
from mixsolver_b200 import solver as S

PRECISION = {"fp64": abi.PREC_FP64, "mixed": abi.PREC_MIXED}


def listed():
    return [
        # The reference's own size of problem, in its own arithmetic: a 64 x 64 lid-driven
        # cavity, IC(0) and ILU(0), where launches and sweeps decide.
        {"name": "cavity2d_64_fp64", "kind": "cavity2d", "n": 64, "precision": "fp64", "steps": 4},
        # The reference's published transient cavity: 80 x 80, limited upwind, one PIMPLE
        # time step of 2 outer iterations x 2 corrections.
        {"name": "pimple_80_mixed", "kind": "pimple", "n": 80, "precision": "mixed"},
        # Channel flow in the reference's arithmetic on a grid of blocks.
        {"name": "channel_65k_fp64", "kind": "channel", "nx": 64, "ny": 32, "nz": 32, "precision": "fp64", "steps": 1},
        # A ragged channel, the size of a first coarse run.
        {"name": "channel_42k_mixed", "kind": "channel", "nx": 47, "ny": 29, "nz": 31, "precision": "mixed", "steps": 3},
        # The benchmark's channel.
        {"name": "channel_524k_mixed", "kind": "channel", "nx": 128, "ny": 64, "nz": 64, "precision": "mixed",
         "steps": 2},
        # Buoyant flow with the energy equation, symmetry planes and thermal walls.
        {"name": "thermal_54k_mixed", "kind": "thermal", "nx": 60, "ny": 30, "nz": 30, "precision": "mixed",
         "steps": 2},
        # The largest steady case of the served stream: 126^3 hexahedra.
        {"name": "cavity3d_2M_mixed", "kind": "cavity3d", "n": 126, "precision": "mixed", "steps": 1},
        # A served transient request: one PISO step on hexahedra split into tetrahedra.
        {"name": "piso_83k_mixed", "kind": "piso", "n": 24, "precision": "mixed", "tol": 1e-8},
        # The largest transient case: 3.07 million tetrahedra, solved to 1e-10.
        {"name": "piso_3M_mixed", "kind": "piso", "n": 80, "precision": "mixed", "tol": 1e-10},
        # Many cavities of uneven size advanced together, as a parameter study does.
        {"name": "batch_24_mixed", "kind": "batch", "count": 24, "low": 16, "high": 64, "steps": 2},
        # Stand-alone solves of a variable-coefficient Poisson system held by the host.
        {"name": "system_152k_poly", "kind": "system", "nx": 61, "ny": 53, "nz": 47, "method": "poly"},
        {"name": "system_33k_ic0", "kind": "system", "nx": 32, "ny": 32, "nz": 32, "method": "ic0"},
    ]


def _log(rng, low, high):
    return float(np.exp(rng.uniform(np.log(low), np.log(high))))


def draw(rng):
    """One more case: cell counts spread over their logarithm, odd edges as they come."""
    kind = rng.choice(["cavity2d", "pimple", "channel", "channel", "thermal", "cavity3d", "piso", "piso", "batch",
                       "system"])
    if kind == "cavity2d":
        return {"kind": kind, "n": int(_log(rng, 12, 97)), "precision": rng.choice(["fp64", "mixed"]),
                "steps": rng.randint(2, 5)}
    if kind == "pimple":
        return {"kind": kind, "n": int(_log(rng, 24, 140)), "precision": "mixed"}
    if kind in ("channel", "thermal"):
        fp64 = kind == "channel" and rng.random() < 0.25
        top = 65_000 if fp64 else 520_000 if kind == "channel" else 120_000
        edge = (_log(rng, 4_000, top) / 2.0) ** (1.0 / 3.0)
        return {"kind": kind, "nx": int(2.0 * edge), "ny": max(4, int(edge * rng.uniform(0.8, 1.1))),
                "nz": max(4, int(edge * rng.uniform(0.8, 1.1))), "precision": "fp64" if fp64 else "mixed",
                "steps": rng.randint(1, 2)}
    if kind == "cavity3d":
        return {"kind": kind, "n": int(_log(rng, 4_096, 1_900_000) ** (1.0 / 3.0)), "precision": "mixed", "steps": 1}
    if kind == "piso":
        return {"kind": kind, "n": int((_log(rng, 6_000, 2_500_000) / 6.0) ** (1.0 / 3.0)), "precision": "mixed",
                "tol": rng.choice([1e-8, 1e-10])}
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(5, 24), "low": 16, "high": rng.randint(33, 64), "steps": 2}
    method = rng.choice(["poly", "ic0"])
    edge = _log(rng, 3_000, 200_000 if method == "poly" else 33_000) ** (1.0 / 3.0)
    return {"kind": kind, "nx": int(edge * rng.uniform(0.8, 1.2)), "ny": int(edge * rng.uniform(0.8, 1.2)),
            "nz": int(edge * rng.uniform(0.8, 1.1)), "method": method}


# ---- meshes: read once by a user's program, so made once and kept ----------------


def _renumbered(mesh):
    return cases.rcm_renumber(mesh, S.rcm_order_device)


@functools.lru_cache(maxsize=64)
def _mesh(kind, *size):
    """(mesh, control, geometry) of a flow case."""
    if kind == "cavity2d":
        mesh, ctrl = cases.cavity2d(size[0])
        ctrl.lin_max = 400
    elif kind == "pimple":
        mesh, ctrl = cases.cavity2d(size[0], mu=1e-3, conv_blend=1.0, nonorth=0.0)
        ctrl.transient, ctrl.dt, ctrl.n_time_max = True, 0.01, 10 ** 6
        ctrl.n_outer_iter, ctrl.n_correct, ctrl.lin_max = 2, 2, 300
    elif kind == "channel":
        mesh, ctrl = cases.channel3d(*size, order_fn=S.rcm_order_device)
        ctrl.lin_max = 1000
    elif kind == "thermal":
        # inlet at T = 1.5, outlet with a heat flux, a cold wall, a heated wall, symmetry
        mesh = meshgen.box_hex(*size, lx=2.0, jitter=0.1, seed=31, zones=(4, 5, 6, 7, 8, 8))
        mesh = _renumbered(meshgen.shuffle_cells(mesh, 32))
        _, ctrl = cases.channel3d(4, 2, 2)
        ctrl.mu, ctrl.lin_max = 2e-2, 1000
        b = abi.BcSpec
        ctrl.bcs = [b(zone=4, btype=abi.BC_VINLET, uvel=(0.5, 0.0, 0.0), tval=1.5),
                    b(zone=5, btype=abi.BC_POUTLET, pval=0.0, ttype=2, qval=-0.1),
                    b(zone=6, btype=abi.BC_WALL, ttype=1, tval=0.5),
                    b(zone=7, btype=abi.BC_WALL, ttype=2, qval=0.3),
                    b(zone=8, btype=abi.BC_SYMMETRY)]
        ctrl.energy = ctrl.boussinesq = True
        ctrl.cp, ctrl.k_cond, ctrl.beta, ctrl.tref, ctrl.gravity = 2.0, 0.05, 0.2, 1.0, (0.0, -1.0, 0.0)
    elif kind == "cavity3d":
        mesh, ctrl = cases.cavity3d(size[0], seed=size[0], mom=abi.MOM_JACOBI)
        ctrl.lin_max = 1000
    elif kind == "piso":
        mesh, ctrl = cases.tet_box(size[0], steps=10 ** 6, mom=abi.MOM_JACOBI)
        mesh = _renumbered(mesh)
        ctrl.lin_max = 1000
    else:
        raise ValueError(kind)
    return mesh, ctrl, S.compute_geometry(mesh)


def _size(case):
    return (case["nx"], case["ny"], case["nz"]) if "nx" in case else (case["n"],)


def _edges(case):
    """The cube edges of a batch, log-uniform in cells, uneven and fixed by its size."""
    t = (np.arange(case["count"]) * 0.618034) % 1.0
    return [int(round(case["low"] * (case["high"] / case["low"]) ** v)) for v in t]


# ---- inputs -----------------------------------------------------------------------


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.float64, pin_memory=True).numpy()
    t[...] = a
    return t


def _fields(kind, mesh, geo, rng):
    """A flow under way: the case's mean motion, a seeded smooth disturbance and 1 % noise,
    with the pressure and the face fluxes that go with it."""
    xc = geo["xc"]
    ext = np.maximum(xc.max(0), 1e-12)
    x, y, z = (xc[:, k] / ext[k] for k in range(3))
    if kind == "piso":
        u = meshgen.taylor_green(xc, seed=int(rng.integers(1 << 30)))
    else:
        u = np.zeros((mesh.ncells, 3))
        if kind == "channel":
            u[:, 0] = 24.0 * y * (1 - y) * z * (1 - z) + 0.1
        elif kind == "thermal":
            u[:, 0] = 0.5
        else:
            u[:, 0] = np.sin(np.pi * x) * y * (3 * y - 2)
            u[:, 1] = -0.5 * np.cos(np.pi * x) * y * (1 - y)
        for k in range(2 if kind in ("cavity2d", "pimple") else 3):
            a = rng.uniform(-3.0, 3.0, 3)
            u[:, k] += 0.05 * np.sin(6.0 * (a[0] * x + a[1] * y + a[2] * z) + rng.uniform(0.0, 6.0))
            u[:, k] += 0.01 * rng.standard_normal(mesh.ncells)
    p = 0.05 * np.cos(3.0 * x + rng.uniform(0.0, 6.0)) * np.cos(2.0 * y)
    if kind == "channel":
        p += 0.3 * (1 - x)
    a, b = mesh.c0 - 1, np.maximum(mesh.c1, mesh.c0 * (mesh.c1 == 0)) - 1
    flux = np.einsum("ij,ij->i", 0.5 * (u[a] + u[b]), geo["sf"])
    still = mesh.c1 == 0
    if kind in ("channel", "thermal"):
        still &= ~np.isin(mesh.zone, (4, 5))
    flux[still] = 0.0
    return {"u": _pinned(u), "p": _pinned(p), "flux": _pinned(flux)}


def _poisson(case):
    """Pattern of the 7-point system (1-based CSR) and, per entry, its face or -1 (diagonal)."""
    nx, ny, nz = _size(case)
    n = nx * ny * nz
    c = np.arange(n).reshape(nz, ny, nx)
    lo = np.concatenate([c[:, :, :-1].ravel(), c[:, :-1].ravel(), c[:-1].ravel()])
    hi = np.concatenate([c[:, :, 1:].ravel(), c[:, 1:].ravel(), c[1:].ravel()])
    f = np.arange(lo.size)
    row = np.concatenate([lo, hi, np.arange(n)])
    col = np.concatenate([hi, lo, np.arange(n)])
    face = np.concatenate([f, f, np.full(n, -1)])
    order = np.lexsort((col, row))
    ptr = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(row, minlength=n), out=ptr[1:])
    return lo, hi, (ptr + 1).astype(np.int32), (col[order] + 1).astype(np.int32), face[order], row[order]


_pattern = functools.lru_cache(maxsize=16)(lambda nx, ny, nz: _poisson({"nx": nx, "ny": ny, "nz": nz}))


def _system(case, seed):
    """Matrix values, solution and right-hand side of a seeded system: face coefficients over
    a factor of twenty, a reaction term that keeps it definite, a smooth solution."""
    lo, hi, ptr, col, face, row = _pattern(*_size(case))
    n = ptr.size - 1
    rng = np.random.default_rng(seed)
    k = np.exp(rng.uniform(-1.5, 1.5, lo.size))
    diag = np.bincount(lo, k, n) + np.bincount(hi, k, n) + 1e-3
    val = np.where(face >= 0, -k[np.maximum(face, 0)], diag[row])
    t = np.arange(n) / n
    x = np.sin(9.0 * t + rng.uniform(0.0, 6.0)) + 0.1 * rng.standard_normal(n)
    b = np.bincount(row, val * x[col - 1], n)
    return ptr, col, val, b, x


def prepare(case, seed):
    kind = case["kind"]
    if kind == "system":
        ptr, col, val, b, _ = _system(case, seed)
        return {"kind": kind, "method": case["method"], "args": (ptr, col, val, b, np.zeros_like(b))}
    rng = np.random.default_rng(seed)
    parts = [("cavity3d", (e,)) for e in _edges(case)] if kind == "batch" else [(kind, _size(case))]
    state = {"kind": kind, "steps": case.get("steps", 1), "cases": [], "in": [], "T": None}
    for k, size in parts:
        mesh, ctrl, geo = _mesh(k, *size)
        ctrl = abi.Ctrl(**{**vars(ctrl), "precision": PRECISION[case.get("precision", "mixed")],
                           "lin_tol": case.get("tol", 1e-8)})
        if kind == "batch":
            ctrl.mu = 1.0 / rng.uniform(100.0, 2000.0)
        state["cases"].append(S.UnsCase(mesh, ctrl))
        state["in"].append(_fields(k, mesh, geo, rng))
    if kind == "thermal":
        state["T"] = _pinned(1.0 + 0.3 * np.sin(3.0 * geo["xc"][:, 1]) + 0.01 * rng.standard_normal(mesh.ncells))
    names = ("u", "p", "flux", "gp", "gu", "apc") if kind not in ("piso", "pimple", "batch") else ("u", "p", "flux")
    shapes = S.UnsCase.FIELD_SHAPES
    dims = [{"N": c.N, "F": c.F} for c in state["cases"]]
    # one page-locked array per field, the cases of a batch one after another
    state["out"], state["views"] = {}, [{} for _ in dims]
    for name in names:
        wants = [tuple(d.get(s, s) for s in shapes[name]) for d in dims]
        whole = torch.empty(sum(w[0] for w in wants), *wants[0][1:], dtype=torch.float64, pin_memory=True).numpy()
        at = np.cumsum([0] + [w[0] for w in wants])
        state["out"][name] = whole
        for i, v in enumerate(state["views"]):
            v[name] = whole[at[i]:at[i + 1]]
    if kind == "batch":
        state["batch"] = S.CaseBatch(state["cases"])
    return state


def run(state):
    kind = state["kind"]
    if kind == "system":
        ptr, col, val, b, x0 = state["args"]
        if state["method"] == "poly":
            x, _, _, ierr = S.pcg_poly(ptr, col, val, b, x0, 1e-8, 1000)
        else:
            x, _, _, ierr = S.cg_ic0(ptr, col, val, b, x0, 1e-8, 1000)
        return {"x": x, "ierr": ierr}
    for c, f in zip(state["cases"], state["in"]):
        if kind in ("piso", "pimple"):
            c.upload(u=f["u"], p=f["p"], flux=f["flux"], u_old=f["u"], u_old_old=f["u"])
        else:
            c.upload(u=f["u"], p=f["p"], flux=f["flux"])
    if kind == "batch":
        _, ier = state["batch"].run(0, state["steps"])
        for c, v in zip(state["cases"], state["views"]):
            c.fields(v)
        return {**state["out"], "ier": ier}
    c, view = state["cases"][0], state["views"][0]
    if kind in ("piso", "pimple"):
        ier, _ = c.piso_run(1, logcap=4) if kind == "piso" else c.pimple_run(1, logcap=4)
        c.fields(view)
        return {**state["out"], "ier": ier}
    if state["T"] is not None:
        c.upload_T(state["T"])
    ier, _, _ = c.simple_run_fields(state["steps"], out=view, logcap=16)
    res = {**state["out"], "ier": ier}
    if state["T"] is not None:
        res["T"] = c.temperature()[0]
    return res


def _counts(case):
    """(cells, faces) of all the meshes of a case."""
    kind = case["kind"]
    if kind in ("cavity2d", "pimple"):
        n = case["n"]
        return n * n, 2 * n * (n - 1) + 4 * n + 2 * n * n
    if kind == "piso":
        n = case["n"]
        return 6 * n ** 3, 12 * n ** 3 + 6 * n * n
    boxes = [(e, e, e) for e in _edges(case)] if kind == "batch" else [
        _size(case) if "nx" in case else (case["n"],) * 3]
    return (sum(a * b * c for a, b, c in boxes),
            sum(3 * a * b * c + a * b + b * c + a * c for a, b, c in boxes))


def work(case):
    """The least a pass can do: the fields up and down once, the mesh's face and cell arrays
    read once an outer iteration, and one multiplication by the matrix a linear system."""
    if case["kind"] == "system":
        nx, ny, nz = _size(case)
        n = nx * ny * nz
        nnz = 7 * n
        return {"bytes": 12.0 * nnz + 4.0 * n + 24.0 * n, "flops": 2.0 * nnz}
    cells, faces = _counts(case)
    steps = {"piso": 1, "pimple": 2}.get(case["kind"], case.get("steps", 1))
    solves = 5 if case["kind"] in ("piso", "pimple", "thermal") else 4
    up = 8.0 * (4 * cells + faces)
    down = up + (0.0 if case["kind"] in ("piso", "pimple", "batch") else 8.0 * 13 * cells)
    mesh = faces * (3 * 4 + 8.0 * 11) + cells * 8.0 * 8
    return {"bytes": up + down + steps * mesh,
            "flops": steps * (300.0 * faces + solves * 2.0 * (cells + 2.0 * faces))}


def exact(case, seed):
    """The solution a system was made from; a whole flow step has no value apart from its solver's."""
    if case["kind"] != "system":
        return None
    return {"x": _system(case, seed)[4], "ierr": None}
