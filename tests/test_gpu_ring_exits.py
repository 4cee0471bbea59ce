"""CTAs of a split default sweep that give up waiting leave with nothing in
flight to them.

Results reach the other CTAs of a cluster as asynchronous stores. When a
bounded wait runs out, the CTA must send nothing more (later levels' bytes
would pile up on the others' barriers, which count to 2^20 - 1) and must not
end before what was sent to it has landed. Two ways to give up, neither of
which faults or hangs: CTA rank 1 sends nothing, so that every CTA of the
cluster gives up at its second or third level; and a bound of 1 ns, so that
any wait which is not met at once gives up, somewhere along the sweep. The
sweep counts the CTAs that gave up and those that saw every byte land: the
two must be equal, the status must report the timeout, and with the bound
restored the same objects apply as before, bit for bit.
"""
import ctypes as C

import numpy as np
import pytest

from gpu_fem_b200 import mesh as M

pytestmark = pytest.mark.gpu

# separate plates, nx, ny, fill level, rows of a strip one element wide: two
# CTAs, four CTAs, levels of one row at both ends of the sweep, and a triangle of
# 80,601 rows (its later levels are more than a barrier can count)
FULL = 0x7FFFFFFF
CASES = {"two": (2, 100, 6, FULL, 0), "four": (1, 256, 128, 6, 0), "tail": (1, 200, 60, 8, 20),
         "long": (1, 400, 200, 2, 0)}


def _factored(case, precision):
    import torch
    from gpu_fem_b200.assembler import ElementAssembler, ILUk_Preconditioner, createBsrMat
    parts, nx, ny, fill, tail = CASES[case]
    m = M.plate(nx, ny + tail, 1.0, 0.5, lambda x, y: 0.006 + 0 * x, "x0",
                lambda q: 1e3 + 0 * q[:, 0])
    if tail:  # beyond row ny only the last column of elements
        e = np.arange(m.conn.shape[0])
        keep = (e // nx < ny) | (e % nx == nx - 1)
        m.conn, m.thick = m.conn[keep], m.thick[keep]
        nodes = np.unique(m.conn)
        new = np.full(m.num_nodes, -1)
        new[nodes] = np.arange(len(nodes))
        bcs = m.bcs[new[m.bcs // 6] >= 0]
        m.bcs = (6 * new[bcs // 6] + bcs % 6).astype(np.int32)
        m.conn, m.xpts = new[m.conn].astype(np.int32), m.xpts[nodes]
    n = m.num_nodes
    m = M.ShellMesh(np.concatenate([m.conn + k * n for k in range(parts)]).astype(np.int32),
                    np.concatenate([m.xpts + [0.0, 2.0 * k, 0.0] for k in range(parts)]),
                    np.tile(m.thick, parts),
                    np.concatenate([m.bcs + 6 * n * k for k in range(parts)]).astype(np.int32),
                    np.zeros(6 * n * parts))
    A = ElementAssembler.from_mesh(m, ordering="natural")
    K = createBsrMat(A)
    A.add_jacobian(None, K, fuse_bcs=True)
    P = ILUk_Preconditioner(A, fill, precision)
    P.factor(K)
    torch.cuda.synchronize()
    return m, P


@pytest.mark.parametrize("case", list(CASES))
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_ctas_that_give_up_leave_quietly(case, precision):
    import torch
    from gpu_fem_b200 import _lib as L
    lib = L.lib()
    m, P = _factored(case, precision)
    lay = P.sweep_layout()
    ctas = lay["L"][1] + lay["U"][1]
    assert ctas == (4 if case == "two" else 8), lay

    def exits():
        g, q = C.c_int32(), C.c_int32()
        L.check(lib.gf_test_sweep_exits(P.h, C.byref(g), C.byref(q)), "exits")
        return g.value, q.value

    r = torch.tensor(np.random.default_rng(3).standard_normal(m.num_dof), device="cuda")
    z0, z1 = torch.zeros_like(r), torch.zeros_like(r)
    P.apply(r, z0)
    assert P.status() == L.GF_OK and exits() == (0, 0)
    try:
        L.check(lib.gf_test_set_waits(200_000, 1), "set_waits")
        P.apply(r, z1)
        assert P.status() == L.GF_TIMEOUT
        gave_up, quiet = exits()
        # every CTA of both sweeps' clusters
        assert gave_up == ctas and quiet == gave_up
        L.check(lib.gf_test_set_waits(1, 0), "set_waits")
        for _ in range(20):
            P.apply(r, z1)
            status = P.status()
            gave_up, quiet = exits()
            assert quiet == gave_up
            assert status == (L.GF_TIMEOUT if gave_up else L.GF_OK)
    finally:
        L.check(lib.gf_test_set_waits(0, 0), "restore waits")
    P.apply(r, z1)
    assert P.status() == L.GF_OK and exits() == (0, 0)
    assert torch.equal(z0, z1)
