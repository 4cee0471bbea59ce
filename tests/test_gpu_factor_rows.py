"""The block ILU factorization at the edges of its row and step layout.

Backward error max |(LU - A) on the pattern| <= 1e-10 max |A| (the gate of the
other factorization tests), where the layout changes: rows with no and with
one lower block, U(k) of up to 4, 16, 32 blocks and more (groups of four in
the update lists, further lists of 32), rows of more than 64 steps and of more
than 80 blocks (updated in global memory), column spans beyond the slot map
(binary searches), and orders that are not ascending.
"""
import numpy as np
import pytest

from gpu_fem_b200 import mesh as M

pytestmark = pytest.mark.gpu

FULL = 0x7FFFFFFF
CASES = {"one_element": (1, 1, 0, "natural"), "strip": (40, 1, 0, "natural"),
         "ilu0": (20, 17, 0, "rcm"), "ilu3": (33, 18, 3, "natural"),
         "ilu10": (40, 33, 10, "natural"), "ilu20": (50, 45, 20, "natural"),
         "full": (30, 18, FULL, "natural"), "long_rows": (100, 90, FULL, "natural"),
         "wide_span": (40, 30, 1, "shuffled")}


@pytest.mark.parametrize("case", list(CASES))
def test_factor_backward_error(case):
    import torch
    from gpu_fem_b200.assembler import ElementAssembler, ILUk_Preconditioner, createBsrMat
    from oracle import pyoracle as po
    nx, ny, fill, order = CASES[case]
    m = M.plate(nx, ny, 1.0, ny / nx, lambda x, y: 0.006 + 0 * x, "all_edges",
                lambda q: 1e3 + 0 * q[:, 0])
    if order == "shuffled":
        new = np.random.default_rng(5).permutation(m.num_nodes)
        m.conn = new[m.conn].astype(np.int32)
        x = np.empty_like(m.xpts)
        x[new] = m.xpts
        m.xpts, order = x, "natural"
        m.bcs = (6 * new[m.bcs // 6] + m.bcs % 6).astype(np.int32)
    A = ElementAssembler.from_mesh(m, ordering=order)
    K = createBsrMat(A)
    A.add_jacobian(None, K, fuse_bcs=True)
    P = ILUk_Preconditioner(A, fill, "fp64")
    bd = A.getBsrData()
    first = None
    for _ in range(2):  # a second factorization on the same buffers, bitwise
        P.factor(K)
        torch.cuda.synchronize()
        r, c, lu = P.get()
        assert first is None or np.array_equal(first.view(np.uint64), lu.view(np.uint64))
        first = lu
    Ak = po.scatter_to_pattern(bd["rowPtr"], bd["colPtr"], K.values_host(), r, c)
    err, amax = po.ilu_backward_error(r, c, lu, Ak, dinv=True)
    assert err <= 1e-10 * amax, (err, amax)
