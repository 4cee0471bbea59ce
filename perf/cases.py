"""Performance cases of the shell-analysis path.

Each case is one call (or the few calls that always go together) that a user
of the framework makes: assembling a Jacobian or a residual, a BSR product, a
numeric ILU(k) factorization, a preconditioner apply, one linear solve, a
batch of design variants, the complete direct solve. Sizes come from the
framework's own meshes: the 10x10 plate, the 400x200 plate, the 300x300 plate,
the stiffened box, the 64 plates of the batch workload (grids 16^2 to 256^2,
aspect 1 to 4, t 2 to 8 mm) and the serving size classes, with odd sizes
between them.

`prepare` makes the mesh, the material and load fields, the displacement or
right-hand-side vectors and the handles that a program keeps (assembler,
matrix, preconditioner, batch); the seed moves nodes, thicknesses, loads and
vectors, never the sizes. `exact` restates the element (MITC4 shell, strain-
displacement form), the Dirichlet rows and columns, the block ILU(k) and the
solve in plain torch / numpy in 64 bits.
"""
from __future__ import annotations

import math
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

from gpu_fem_b200 import mesh as M
from gpu_fem_b200.assembler import (BsrMat, DeviceVec, ElementAssembler, ILUk_Preconditioner,
                                    SolveOptions, direct_solve, gmres_solve)
from gpu_fem_b200.batch import Batch, solve_opts

# ILU fill level of each of the 64 plates of the batch workload, as the batch
# benchmark runs them (every plate converges with these to 1e-8).
BATCH64_FILLS = (12, 16, 12, 7, 6, 6, 10, 8, 8, 5, 8, 6, 10, 6, 12, 12, 8, 8, 8, 12, 12, 6, 10, 10,
                 6, 16, 12, 6, 7, 8, 10, 12, 5, 12, 5, 10, 7, 6, 5, 12, 16, 16, 5, 12, 6, 10, 10,
                 12, 10, 12, 8, 7, 16, 8, 6, 5, 8, 10, 12, 16, 4, 4, 10, 12)


def listed():
    return [
        # the smallest Jacobian a user assembles (quick-start plate): launches count
        {"name": "jacobian_10x10", "kind": "jacobian", "nx": 10, "ny": 10},
        # one Newton / design step's Jacobian and residual on the scale plate
        {"name": "jacobian_400x200", "kind": "jacobian", "nx": 400, "ny": 200},
        # residual check of a displacement field, the reference's 300x300 plate
        {"name": "residual_300x300", "kind": "residual", "nx": 300, "ny": 300},
        # the matrix-vector product of a user's own Krylov loop
        {"name": "spmv_400x200", "kind": "spmv", "nx": 400, "ny": 200},
        # refactoring after a design change and applying once: an odd small
        # plate in FP64, and a large plate with FP32 factors
        {"name": "factor_61x37_fp64", "kind": "factor", "nx": 61, "ny": 37, "fill": 8,
         "precision": "fp64", "ordering": "natural"},
        {"name": "factor_256x128_fp32", "kind": "factor", "nx": 256, "ny": 128, "fill": 6,
         "precision": "fp32", "ordering": "natural"},
        # one preconditioner apply inside a user's own Krylov loop
        {"name": "apply_256x128_fp32", "kind": "apply", "nx": 256, "ny": 128, "fill": 6,
         "precision": "fp32", "ordering": "natural"},
        {"name": "apply_box_72x18x6_fp64", "kind": "apply", "box": True, "nx": 72, "ny": 18,
         "nz": 6, "fill": 12, "precision": "fp64", "ordering": "rcm"},
        # one right-hand side on a small odd plate, everything in FP64
        {"name": "solve_33x21_fp64", "kind": "solve", "nx": 33, "ny": 21, "fill": 8,
         "precision": "fp64", "ordering": "natural"},
        # a serving slot group: eight design variants of the smallest size
        # class (5e3 DOF), assembled, factored (FP32) and solved together
        {"name": "batch_8x_28x28", "kind": "batch", "plates": 8, "nx": 28, "ny": 28, "fill": 12,
         "precision": "fp32"},
        # the batch workload: 64 uneven plates, assembled, factored and solved
        {"name": "batch_64_plates", "kind": "batch64", "precision": "fp32"},
        # the complete block LU solve, symbolic setup included
        {"name": "direct_40x20", "kind": "direct", "nx": 40, "ny": 20},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["jacobian", "jacobian", "residual", "spmv", "factor", "factor", "apply",
                       "apply", "solve", "solve", "batch", "batch", "direct"])
    if kind in ("jacobian", "residual", "spmv"):
        nx = _log(rng, 7, 400)
        return {"kind": kind, "nx": nx, "ny": max(5, int(nx / rng.uniform(1.0, 4.0)))}
    if kind == "direct":
        ny = rng.randint(6, 20)
        return {"kind": kind, "nx": rng.randint(ny, 40), "ny": ny}
    if kind == "batch":
        nx = rng.randint(16, 60)
        return {"kind": kind, "plates": rng.randint(2, 12), "nx": nx,
                "ny": max(16, int(nx / rng.uniform(1.0, 3.0))), "fill": rng.choice([12, 14, 16]),
                "precision": rng.choice(["fp32", "fp32", "fp64"])}
    # fills from where the block ILU of these plates is stable (lower ones
    # need a thicker or finer plate); RCM on the smaller plates
    rcm = rng.random() < 0.25
    nx = _log(rng, 20, 90 if rcm else 200)
    return {"kind": kind, "nx": nx, "ny": max(16, int(nx / rng.uniform(1.0, 3.0))),
            "fill": rng.choice([12, 14] if rcm else [8, 9, 10, 12]),
            "precision": rng.choice(["fp64", "fp32"]),
            "ordering": "rcm" if rcm else "natural"}


# ------------------------------------------------------------------ inputs
def _mesh(case, seed):
    """The case's mesh with the seed's nodes, thickness field and load."""
    rs = np.random.RandomState(seed)
    nx, ny = case["nx"], case["ny"]
    if case.get("box"):
        m = M.box(nx, ny, case["nz"])
        m.thick *= rs.uniform(1.0, 1.15, m.num_elements)
        m.loads *= rs.uniform(0.5, 2.0)
        return m
    p0, kx = rs.uniform(0.5e3, 2e3), rs.uniform(0.5, 2.0)
    shell = case["kind"] in ("jacobian", "residual", "spmv")
    # clamped plate with unit length, square elements, jittered nodes
    m = M.plate(nx, ny, 1.0, ny / nx, lambda x, y: 0.005 + 0 * x, "all_edges",
                lambda q: p0 * (1.0 + 0.3 * np.sin(kx * np.pi * q[:, 0])),
                jitter=0.1 if shell else 0.02, seed=seed + 1)
    m.thick *= rs.uniform(1.0, 1.3, m.num_elements)
    if shell:  # a shallow doubly curved panel
        m.xpts[:, 2] = 0.05 * np.sin(np.pi * m.xpts[:, 0]) * np.cos(kx * m.xpts[:, 1])
    return m


def _batch64_meshes(seed):
    rs = np.random.RandomState(seed)
    meshes = M.batch_config4(64)
    for m in meshes:
        m.thick *= rs.uniform(1.0, 1.1)
        m.loads *= rs.uniform(0.5, 2.0)
    return meshes


def _vector(n, seed):
    return torch.tensor(np.random.RandomState(seed + 7).standard_normal(n), device="cuda")


class _Values:
    """Device view of a matrix's block values."""

    def __init__(self, mat):
        self.mat = mat
        self.__cuda_array_interface__ = {"shape": (36 * mat.nnzb,), "typestr": "<f8",
                                         "data": (mat.getPtr(), False), "version": 2}


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind}
    if kind in ("batch", "batch64"):
        if kind == "batch64":
            meshes, fills = _batch64_meshes(seed), BATCH64_FILLS
        else:
            meshes = [_mesh(case, seed + 1000 * k) for k in range(case["plates"])]
            fills = [case["fill"]] * len(meshes)
        with ThreadPoolExecutor(max_workers=8) as ex:
            asms = list(ex.map(lambda m: ElementAssembler.from_mesh(m, ordering="natural"), meshes))
            pcs = list(ex.map(lambda j: ILUk_Preconditioner(j[0], j[1], case["precision"]),
                              zip(asms, fills)))
        mats = [BsrMat(a) for a in asms]
        s["batch"] = Batch(asms, mats, pcs)
        s["b"] = [torch.tensor(m.loads, device="cuda") for m in meshes]
        s["x"] = [torch.zeros_like(b) for b in s["b"]]
        s["opts"] = solve_opts(1e-8)
        return s
    m = _mesh(case, seed)
    A = ElementAssembler.from_mesh(m, ordering=case.get("ordering", "natural"))
    s["A"] = A
    n = m.num_dof
    if kind == "residual":
        s["u"] = DeviceVec(1e-3 * _vector(n, seed))
        s["res"] = DeviceVec(n)
        return s
    s["K"] = K = BsrMat(A)
    if kind == "jacobian":
        A.set_variables(DeviceVec(1e-3 * _vector(n, seed)))
        s["res"] = DeviceVec(n)
        s["values"] = torch.as_tensor(_Values(K), device="cuda")
        return s
    A.add_jacobian(None, K, fuse_bcs=True)
    if kind == "spmv":
        s["v"], s["y"] = _vector(n, seed), torch.zeros(n, dtype=torch.float64, device="cuda")
        return s
    s["b"] = torch.tensor(m.loads, device="cuda")
    s["x"] = torch.zeros_like(s["b"])
    if kind == "direct":
        return s
    s["P"] = P = ILUk_Preconditioner(A, case["fill"], case["precision"])
    if kind != "factor":
        P.factor(K)
    s["r"], s["z"] = _vector(n, seed), torch.zeros(n, dtype=torch.float64, device="cuda")
    s["opts"] = SolveOptions(rtol=1e-8, restart=100)
    return s


def run(s):
    kind = s["kind"]
    if kind == "jacobian":
        s["A"].add_jacobian(s["res"], s["K"], fuse_bcs=True)
        return {"K": s["values"], "res": s["res"].t}
    if kind == "residual":
        s["A"].set_variables(s["u"])
        s["A"].add_residual(s["res"])
        return s["res"].t
    if kind == "spmv":
        s["K"].spmv(s["v"], s["y"])
        return s["y"]
    if kind == "factor":
        s["P"].factor(s["K"])
        s["P"].apply(s["r"], s["z"])
        return s["z"]
    if kind == "apply":
        s["P"].apply(s["r"], s["z"])
        return s["z"]
    if kind == "solve":
        s["x"].zero_()
        gmres_solve(s["A"], s["K"], s["P"], s["b"], s["x"], s["opts"])
        return s["x"]
    if kind == "direct":
        direct_solve(s["A"], s["K"], s["b"], s["x"])
        return s["x"]
    s["batch"].assemble()
    s["batch"].factor()
    for x in s["x"]:
        x.zero_()
    s["batch"].solve(s["b"], s["x"], s["opts"])
    return s["x"]


# -------------------------------------------------------------------- work
def _grid(case):
    """Nodes, elements and matrix blocks (node pairs sharing an element)."""
    nx, ny = case["nx"], case["ny"]
    if case.get("box"):
        nz = case["nz"]
        ne = 2 * nx * ny + 2 * nx * nz + 10 * ny * nz
        nn = (2 * (nx + 1) * (ny + 1) + 2 * (nx + 1) * (nz - 1)) + 10 * (ny - 1) * (nz - 1)
        return nn, ne, 9 * nn
    return (nx + 1) * (ny + 1), nx * ny, (3 * nx + 1) * (3 * ny + 1)


def _ilu_blocks(nn, fill):
    """Blocks of the ILU(k) factor of a gridded shell: about 2 (2 k + 2) + 1 a
    row (k + 1 along the line and k + 2 in the neighbouring line, each side)."""
    return nn * (2 * (2 * fill + 3) + 1)


def work(case):
    """One pass: inputs read once, results written once; operations of the
    element products (B^T D B: 36 x 24 x 24 multiply-adds; B^T D B u for the
    residual), of the block updates and of the products."""
    kind = case["kind"]
    if kind == "batch64":
        parts = [dict(case, kind="plate", nx=m.meta["nxe"], ny=m.meta["nye"], fill=k)
                 for m, k in zip(M.batch_config4(64), BATCH64_FILLS)]
    elif kind == "batch":
        parts = [case] * case["plates"]
    else:
        parts = [case]
    byt = flo = 0.0
    for c in parts:
        nn, ne, nnzb = _grid(c)
        asm = 24.0 * ne + nn * (24 + 48) + 288.0 * nnzb
        asm_f = 2.0 * 36 * 24 * 24 * ne
        vs = 4 if case.get("precision") == "fp32" else 8
        fb = _ilu_blocks(nn, c.get("fill", 0))
        low = (fb / nn - 1) / 2
        fac = 288.0 * nnzb + 36.0 * vs * fb
        fac_f = 2.0 * 216 * nn * low * (low + 1) / 2
        app = (36.0 * vs + 4) * fb + 96.0 * nn
        app_f = 72.0 * fb
        mul = (288.0 + 4) * nnzb + 96.0 * nn
        mul_f = 72.0 * nnzb
        if kind == "jacobian":
            byt, flo = byt + asm + 48.0 * nn, flo + asm_f
        elif kind == "residual":
            byt, flo = byt + 24.0 * ne + nn * (24 + 96 + 48), flo + 2.0 * 2 * 36 * 24 * ne
        elif kind == "spmv":
            byt, flo = byt + mul, flo + mul_f
        elif kind == "factor":
            byt, flo = byt + fac + app, flo + fac_f + app_f
        elif kind == "apply":
            byt, flo = byt + app, flo + app_f
        elif kind == "direct":
            bw = min(c["nx"], c["ny"]) + 2  # banded complete factor
            byt += 288.0 * nnzb + 2 * 288.0 * nn * bw
            flo += 2.0 * 216 * nn * bw * bw
        else:
            # a solve: about 20 steps of apply, product and two passes over
            # the basis (solve_33x21: about 10)
            its = 10 if kind == "solve" else 20
            vec = 2 * 48.0 * nn * its / 2
            byt += its * (app + mul + vec)
            flo += its * (app_f + mul_f + 4 * 6.0 * nn * its / 2)
            if kind != "solve":
                byt, flo = byt + asm + fac, flo + asm_f + fac_f
    return {"bytes": byt, "flops": flo}


# ------------------------------------------------------------ 64-bit results
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _shape(xi, eta, dev):
    s = torch.tensor([-1.0, 1.0, -1.0, 1.0], dtype=torch.float64, device=dev)
    t = torch.tensor([-1.0, -1.0, 1.0, 1.0], dtype=torch.float64, device=dev)
    fx, fe = 0.5 * (1 + s * xi), 0.5 * (1 + t * eta)
    return fx * fe, 0.5 * s * fe, 0.5 * t * fx


def _frame(Xxi, n0):
    """Columns (t1, n x t1, n): t1 = dX/dxi projected off the normal."""
    n = n0 / n0.norm(dim=-1, keepdim=True)
    t1 = Xxi - (Xxi * n).sum(-1, keepdim=True) * n
    t1 = t1 / t1.norm(dim=-1, keepdim=True)
    return torch.stack([t1, torch.linalg.cross(n, t1), n], dim=-1)


def _strain_matrices(X):
    """B (element, point, 9, 24) and det Xd (element, point) of the MITC4
    shell: E = (membrane 3, bending 3, transverse shear 2, drilling 1) = B u."""
    dev, ne = X.device, X.shape[0]
    f64 = dict(dtype=torch.float64, device=dev)
    field = lambda w, f: torch.einsum("n,enk->ek", w, f)  # noqa: E731
    nodes = [(-1.0, -1.0), (1.0, -1.0), (-1.0, 1.0), (1.0, 1.0)]
    fn = []
    for xi, eta in nodes:
        _, Nx, Ne = _shape(xi, eta, dev)
        c = torch.linalg.cross(field(Nx, X), field(Ne, X))
        fn.append(c / c.norm(dim=-1, keepdim=True))
    fn = torch.stack(fn, 1)
    # director of DOF (a, 3 + k): e_k x fn_a
    eye = torch.eye(3, **f64)
    V = torch.linalg.cross(eye[None, None].expand(ne, 4, 3, 3), fn[:, :, None].expand(ne, 4, 3, 3))

    def in_plane(xi, eta, p, q):
        """Tensor strain component (p, q) of the tying points from the
        gradients in directions p, q (0: xi, 1: eta)."""
        N, *d = _shape(xi, eta, dev)
        g = [field(d[0], X), field(d[1], X)]
        row = torch.zeros(ne, 4, 6, **f64)
        row[:, :, :3] = 0.5 * (d[p][None, :, None] * g[q][:, None] + d[q][None, :, None] * g[p][:, None])
        return row.reshape(ne, 24)

    def transverse(xi, eta, p):
        N, *d = _shape(xi, eta, dev)
        g, n0 = field(d[p], X), field(N, fn)
        row = torch.zeros(ne, 4, 6, **f64)
        row[:, :, :3] = 0.5 * d[p][None, :, None] * n0[:, None]
        row[:, :, 3:] = 0.5 * N[None, :, None] * torch.einsum("ek,eack->eac", g, V)
        return row.reshape(ne, 24)

    t11 = [in_plane(0.0, e, 0, 0) for e in (-1.0, 1.0)]
    t22 = [in_plane(x, 0.0, 1, 1) for x in (-1.0, 1.0)]
    t12 = in_plane(0.0, 0.0, 0, 1)
    t23 = [transverse(x, 0.0, 1) for x in (-1.0, 1.0)]
    t13 = [transverse(0.0, e, 0) for e in (-1.0, 1.0)]
    drill = []
    for n, (xi, eta) in enumerate(nodes):
        _, Nx, Ne = _shape(xi, eta, dev)
        T = _frame(field(Nx, X), fn[:, n])
        XT = torch.linalg.solve(torch.stack([field(Nx, X), field(Ne, X), fn[:, n]], -1), T)
        grad = Nx[None, :, None] * XT[:, None, 0, :2] + Ne[None, :, None] * XT[:, None, 1, :2]
        row = torch.zeros(ne, 4, 6, **f64)
        row[:, :, :3] = 0.5 * (T[:, None, :, 1] * grad[:, :, None, 0] - T[:, None, :, 0] * grad[:, :, None, 1])
        row[:, n, 3:] = -torch.linalg.cross(T[:, :, 0], T[:, :, 1])
        drill.append(row.reshape(ne, 24))
    B, det = torch.zeros(ne, 4, 9, 24, **f64), torch.zeros(ne, 4, **f64)
    r3 = 0.577350269189626
    for q in range(4):
        xi, eta = (-r3, r3)[q % 2], (-r3, r3)[q // 2]
        N, Nx, Ne = _shape(xi, eta, dev)
        n0, z = field(N, fn), torch.zeros(ne, 3, **f64)
        Xd = torch.stack([field(Nx, X), field(Ne, X), n0], -1)
        Xz = torch.stack([field(Nx, fn), field(Ne, fn), z], -1)
        T = _frame(Xd[..., 0], n0)
        Xi = torch.linalg.inv(Xd)
        A = Xi @ T
        Az = -Xi @ Xz @ A
        det[:, q] = torch.linalg.det(Xd)
        a, b = (0.5 * (1 - eta), 0.5 * (1 + eta)), (0.5 * (1 - xi), 0.5 * (1 + xi))
        G = torch.zeros(ne, 3, 3, 24, **f64)
        G[:, 0, 0] = a[0] * t11[0] + a[1] * t11[1]
        G[:, 1, 1] = b[0] * t22[0] + b[1] * t22[1]
        G[:, 0, 1] = G[:, 1, 0] = t12
        G[:, 1, 2] = G[:, 2, 1] = b[0] * t23[0] + b[1] * t23[1]
        G[:, 0, 2] = G[:, 2, 0] = a[0] * t13[0] + a[1] * t13[1]
        e = torch.einsum("eia,eijl,ejb->eabl", A, G, A)
        # displacement gradients: mid-surface through Az, director through A and Az
        D = torch.stack([Nx, Ne, torch.zeros_like(N)], -1)
        D1 = torch.stack([Nx, Ne, N], -1)
        u1 = torch.zeros(ne, 3, 3, 4, 6, **f64)
        g0 = torch.einsum("ni,eib->enb", D, Az)
        g1 = torch.einsum("ni,eib->enb", D[:, :2], A[:, :2]) + torch.einsum("n,eb->enb", N, Az[:, 2])
        for c in range(3):
            u1[..., c] = torch.einsum("ea,enb->eabn", T[:, c], g0)
            w = torch.einsum("eia,eni->ena", T, V[:, :, c])
            u1[..., 3 + c] = torch.einsum("ena,enb->eabn", w, g1)
        u1 = u1.reshape(ne, 3, 3, 24)
        B[:, q, 0], B[:, q, 1], B[:, q, 2] = e[:, 0, 0], e[:, 1, 1], 2 * e[:, 0, 1]
        B[:, q, 3], B[:, q, 4], B[:, q, 5] = u1[:, 0, 0], u1[:, 1, 1], u1[:, 0, 1] + u1[:, 1, 0]
        B[:, q, 6], B[:, q, 7] = 2 * e[:, 1, 2], 2 * e[:, 0, 2]
        B[:, q, 8] = sum(N[n] * drill[n] for n in range(4))
    return B, det


def _stress_matrix(thick, E, nu):
    """D (element, 9, 9) of the isotropic shell, mid-surface reference."""
    D = torch.zeros(thick.shape[0], 9, 9, dtype=torch.float64, device=thick.device)
    c, g = E / (1 - nu * nu), E / 2 / (1 + nu)
    for o, w in ((0, thick), (3, thick ** 3 / 12)):
        D[:, o, o] = D[:, o + 1, o + 1] = c * w
        D[:, o, o + 1] = D[:, o + 1, o] = nu * c * w
        D[:, o + 2, o + 2] = g * w
    D[:, 6, 6] = D[:, 7, 7] = 5.0 / 6.0 * g * thick
    D[:, 8, 8] = 10.0 * 5.0 / 6.0 * g * thick
    return D


def _elements(m):
    """K_e (element, 24, 24) and the DOF of each element column."""
    dev = _device()
    X = torch.tensor(m.xpts[m.conn], device=dev)
    out = []
    for lo in range(0, m.num_elements, 20000):
        B, det = _strain_matrices(X[lo:lo + 20000])
        D = _stress_matrix(torch.tensor(m.thick[lo:lo + 20000], device=dev), m.E, m.nu)
        out.append(torch.einsum("eqil,eij,eqjk,eq->elk", B, D, B, det))
    conn = torch.tensor(m.conn, dtype=torch.int64, device=dev)
    dof = (6 * conn[:, :, None] + torch.arange(6, device=dev)).reshape(-1, 24)
    return torch.cat(out), dof


def _free(m, dev):
    f = torch.ones(m.num_dof, dtype=torch.float64, device=dev)
    f[torch.tensor(m.bcs, dtype=torch.int64, device=dev)] = 0.0
    return f


def _product(Ke, dof, v):
    y = torch.zeros_like(v)
    return y.index_add(0, dof.reshape(-1), torch.einsum("elk,ek->el", Ke, v[dof]).reshape(-1))


def _pattern(m):
    """Sorted block columns of every node row (natural order)."""
    c = m.conn.astype(np.int64)
    keys = np.unique((c[:, :, None] * m.num_nodes + c[:, None, :]).ravel())
    return keys


def _blocks(m):
    """Block values (block, 6, 6) in row-sorted order, Dirichlet rows and
    columns applied, and the sorted keys row * nodes + column."""
    Ke, dof = _elements(m)
    dev, n = Ke.device, m.num_nodes
    keys = torch.tensor(_pattern(m), device=dev)
    conn = torch.tensor(m.conn, dtype=torch.int64, device=dev)
    where = torch.searchsorted(keys, (conn[:, :, None] * n + conn[:, None, :]).reshape(-1))
    vals = torch.zeros(keys.numel(), 6, 6, dtype=torch.float64, device=dev)
    vals.index_add_(0, where, Ke.reshape(-1, 4, 6, 4, 6).permute(0, 1, 3, 2, 4).reshape(-1, 6, 6))
    free = _free(m, dev).reshape(n, 6)
    r, c = keys // n, keys % n
    vals *= free[r][:, :, None] * free[c][:, None, :]
    d = torch.nonzero(r == c).reshape(-1)
    i6 = torch.arange(6, device=dev)
    vals[d[:, None], i6, i6] += 1.0 - free[r[d]]
    return vals, keys, Ke, dof


def _iluk(n, vals, keys, fill, r):
    """z = U^-1 L^-1 r of the block ILU(k) factor on the level-of-fill pattern."""
    vals, keys = vals.cpu().numpy(), keys.cpu().numpy()
    rows = [dict() for _ in range(n)]
    a = [dict() for _ in range(n)]
    for q, k in enumerate(keys):
        rows[k // n][int(k % n)] = 0
        a[k // n][int(k % n)] = q
    up, fac, dinv = [None] * n, [None] * n, [None] * n
    for i in range(n):
        lev, todo = rows[i], sorted(j for j in rows[i] if j < i)
        t = 0
        while t < len(todo):
            k, lk = todo[t], lev[todo[t]]
            for j, lj in up[k]:
                v = lk + lj + 1
                if v <= fill and v < lev.get(j, 1 << 30):
                    if j not in lev and j < i:
                        todo.append(j)
                        todo[t + 1:] = sorted(todo[t + 1:])
                    lev[j] = v
            t += 1
        cols = sorted(lev)
        up[i] = [(j, lev[j]) for j in cols if j > i]
        R = np.zeros((len(cols), 6, 6))
        pos = {j: p for p, j in enumerate(cols)}
        for j, q in a[i].items():
            R[pos[j]] = vals[q]
        for k in (j for j in cols if j < i):
            ck, Rk, dk = fac[k]
            L = R[pos[k]] @ dinv[k]
            R[pos[k]] = L
            hit = [(pos[j], p) for p, j in enumerate(ck[dk + 1:], dk + 1) if j in pos]
            if hit:
                to, fr = zip(*hit)
                R[list(to)] -= L @ Rk[list(fr)]
        dinv[i] = np.linalg.inv(R[pos[i]])
        fac[i] = (cols, R, pos[i])
    z = r.reshape(n, 6).copy()
    for i in range(n):
        cols, R, d = fac[i]
        if d:
            z[i] -= np.einsum("kij,kj->i", R[:d], z[cols[:d]])
    for i in range(n - 1, -1, -1):
        cols, R, d = fac[i]
        t = z[i]
        if d + 1 < len(cols):
            t = t - np.einsum("kij,kj->i", R[d + 1:], z[cols[d + 1:]])
        z[i] = dinv[i] @ t
    return z.reshape(-1)


def _dense_solution(m):
    """K x = b by a dense 64-bit factorization, refined once."""
    vals, keys, _, _ = _blocks(m)
    n, dev = m.num_nodes, vals.device
    K = torch.zeros(n, 6, n, 6, dtype=torch.float64, device=dev)
    K[keys // n, :, keys % n] = vals
    K = K.reshape(6 * n, 6 * n)
    b = torch.tensor(m.loads, device=dev)[:, None]
    lu = torch.linalg.lu_factor(K)
    x = torch.linalg.lu_solve(*lu, b)
    x = x + torch.linalg.lu_solve(*lu, b - K @ x)
    return x.reshape(-1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch64":
        return None  # up to 3e5 unknowns a problem
    if kind == "batch":
        meshes = [_mesh(case, seed + 1000 * k) for k in range(case["plates"])]
        if max(m.num_dof for m in meshes) > 12000:
            return None
        return [_dense_solution(m) for m in meshes]
    m = _mesh(case, seed)
    if kind == "residual":
        Ke, dof = _elements(m)
        return _product(Ke, dof, 1e-3 * _vector(m.num_dof, seed))
    if kind == "jacobian":
        vals, _, Ke, dof = _blocks(m)
        res = _product(Ke, dof, 1e-3 * _vector(m.num_dof, seed)) * _free(m, Ke.device)
        return {"K": vals.reshape(-1), "res": res}
    if kind == "spmv":
        Ke, dof = _elements(m)
        free, v = _free(m, Ke.device), _vector(m.num_dof, seed)
        return _product(Ke, dof, free * v) * free + (1.0 - free) * v
    if kind in ("solve", "direct"):
        return _dense_solution(m) if m.num_dof <= 20000 else None
    # the preconditioner of the natural order, up to a few thousand rows (the
    # factorization here is a Python loop)
    if case["ordering"] != "natural" or case.get("box") or m.num_nodes * case["fill"] ** 2 > 5e5:
        return None
    vals, keys, _, _ = _blocks(m)
    return _iluk(m.num_nodes, vals, keys, case["fill"], _vector(m.num_dof, seed).cpu().numpy())
