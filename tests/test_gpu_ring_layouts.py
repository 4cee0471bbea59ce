"""Which kernel and which layout of it solves a triangle, and every layout of
the ring sweep against the oracle's triangular solves.

The layouts (CTAs of a cluster, groups of warps) come from a cost model over
rows and blocks a level, so each case states the one it is here for and the
query must report it: one CTA with 2, 3 and 4 groups; two CTAs, which the model
takes for two long rows a level (two separate strips with complete factors);
four CTAs with 2, 3 and 4 groups, one of them on three strips, where one CTA
has no rows at all. The apply agrees with the oracle entry by entry to 1e-12 of
max |z| (the gate of the other sweeps). A numbering whose dependency reach does
not fit the ring is solved by the chunked kernel; in one batch with a plate on
the ring, both problems give bitwise the results they give alone.
"""
import numpy as np
import pytest

from gpu_fem_b200 import mesh as M

pytestmark = pytest.mark.gpu

FULL = 0x7FFFFFFF
# separate plates, nx, ny, fill level -> CTAs, groups of both triangles
CASES = {"c1g2": (1, 48, 40, 16, (1, 2)), "c1g3": (1, 40, 16, 6, (1, 3)),
         "c1g4": (1, 17, 16, 8, (1, 4)), "c2g2": (2, 100, 6, FULL, (2, 2)),
         "c2g3": (2, 80, 6, FULL, (2, 3)), "c4g2": (1, 200, 60, 8, (4, 2)),
         "c4g3": (3, 80, 6, FULL, (4, 3)), "c4g4": (1, 61, 37, 8, (4, 4))}


def _mesh(parts, nx, ny):
    m = M.plate(nx, ny, 1.0, ny / nx, lambda x, y: 0.006 + 0 * x, "all_edges",
                lambda q: 1e3 + 0 * q[:, 0])
    n = m.num_nodes
    return M.ShellMesh(np.concatenate([m.conn + k * n for k in range(parts)]).astype(np.int32),
                       np.concatenate([m.xpts + [0.0, 2.0 * k, 0.0] for k in range(parts)]),
                       np.tile(m.thick, parts),
                       np.concatenate([m.bcs + 6 * n * k for k in range(parts)]).astype(np.int32),
                       np.tile(m.loads, parts))


def _shuffled(nx, ny):
    m = _mesh(1, nx, ny)
    new = np.random.default_rng(5).permutation(m.num_nodes)
    m.conn = new[m.conn].astype(np.int32)
    x, b = np.empty_like(m.xpts), np.empty_like(m.loads)
    x[new] = m.xpts
    b.reshape(-1, 6)[new] = m.loads.reshape(-1, 6)
    m.xpts, m.loads = x, b
    m.bcs = (6 * new[m.bcs // 6] + m.bcs % 6).astype(np.int32)
    return m


def _factored(m, fill, precision, sweep="auto"):
    import torch
    from gpu_fem_b200.assembler import ElementAssembler, ILUk_Preconditioner, createBsrMat
    A = ElementAssembler.from_mesh(m, ordering="natural")
    K = createBsrMat(A)
    A.add_jacobian(None, K, fuse_bcs=True)
    P = ILUk_Preconditioner(A, fill, precision, sweep=sweep)
    P.factor(K)
    torch.cuda.synchronize()
    return A, K, P


@pytest.mark.parametrize("case", list(CASES))
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_every_ring_layout_matches_oracle(case, precision):
    import torch
    from oracle import pyoracle as po
    parts, nx, ny, fill, layout = CASES[case]
    m = _mesh(parts, nx, ny)
    A, K, P = _factored(m, fill, precision)
    assert P.sweep_layout() == {"L": ("ring", *layout), "U": ("ring", *layout)}
    rowp, cols, lu = P.get()
    used = lu.astype(np.float32).astype(np.float64) if precision == "fp32" else lu
    for seed in (1, 2):
        r = np.random.default_rng(seed).standard_normal(m.num_dof)
        z = torch.full((m.num_dof,), float("nan"), dtype=torch.float64, device="cuda")
        P.apply(torch.tensor(r, device="cuda"), z)
        assert P.status() == 0
        ref = po.ilu_apply_dinv(rowp, cols, used, r)
        assert np.abs(z.cpu().numpy() - ref).max() <= 1e-12 * np.abs(ref).max()


def test_other_kernels_are_reported():
    m = _shuffled(90, 90)
    for precision in ("fp64", "fp32"):
        lay = _factored(m, 0, precision)[2].sweep_layout()
        assert lay["L"][0] == lay["U"][0] == "chunked", lay
    m = _mesh(1, 20, 16)
    for sweep, kernel in (("level", "chunked"), ("dataflow", "dataflow")):
        lay = _factored(m, 3, "fp64", sweep)[2].sweep_layout()
        assert lay["L"][0] == lay["U"][0] == kernel, lay


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_both_kernels_in_one_batch(precision):
    import torch
    from gpu_fem_b200.assembler import SolveOptions
    from gpu_fem_b200.batch import Batch
    meshes = [_mesh(1, 61, 37), _shuffled(90, 90), _mesh(1, 17, 16)]
    fills = [8, 0, 8]
    opts = SolveOptions(restart=20, max_iters=20, rtol=1e-30, side=1)

    def solve(which):
        made = [_factored(meshes[k], fills[k], precision) for k in which]
        B = Batch(*map(list, zip(*made)))
        B.factor()
        b = [torch.tensor(meshes[k].loads, device="cuda") for k in which]
        x = [torch.zeros_like(t) for t in b]
        B.solve(b, x, opts)
        return [P.sweep_layout()["L"][0] for _, _, P in made], [t.cpu().numpy() for t in x]

    kernels, together = solve([0, 1, 2])
    assert kernels == ["ring", "chunked", "ring"]
    for k in range(3):
        alone = solve([k])[1][0]
        assert np.abs(alone).max() > 0.0
        assert np.array_equal(alone.view(np.uint64), together[k].view(np.uint64)), k
