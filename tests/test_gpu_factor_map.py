"""The block ILU factorization's column -> slot map on rows of about 256 blocks.

A row keeps a map from its columns to its block slots in shared memory
whenever its columns span at most 1024, however many blocks it has: natural
order plates of 125, 126 and 130 elements in width, whose complete factors have
rows of up to 255, 257 and 265 blocks. The rows that have the map are counted
against the pattern, and the factor's backward error max |(LU - A) on the
pattern| is at most 1e-10 max |A|, the gate of the other factorization tests.
"""
import numpy as np
import pytest

from gpu_fem_b200 import mesh as M

pytestmark = pytest.mark.gpu

FULL = 0x7FFFFFFF


@pytest.mark.parametrize("nx,longest", [(125, 255), (126, 257), (130, 265)])
def test_long_rows_keep_their_column_map(nx, longest):
    import torch
    from gpu_fem_b200.assembler import ElementAssembler, ILUk_Preconditioner, createBsrMat
    from oracle import pyoracle as po
    m = M.plate(nx, 6, 1.0, 0.05, lambda x, y: 0.006 + 0 * x, "all_edges",
                lambda q: 1e3 + 0 * q[:, 0])
    A = ElementAssembler.from_mesh(m, ordering="natural")
    K = createBsrMat(A)
    A.add_jacobian(None, K, fuse_bcs=True)
    P = ILUk_Preconditioner(A, FULL, "fp64")
    P.factor(K)
    torch.cuda.synchronize()
    bd = A.getBsrData()
    r, c, lu = P.get()
    n = np.diff(r)
    assert n.max() == longest
    span = c[r[1:] - 1] - c[r[:-1]] + 1
    assert P.factor_layout() == {"staged": int((n <= 80).sum()), "mapped": int((span <= 1024).sum())}
    Ak = po.scatter_to_pattern(bd["rowPtr"], bd["colPtr"], K.values_host(), r, c)
    err, amax = po.ilu_backward_error(r, c, lu, Ak, dinv=True)
    assert err <= 1e-10 * amax, (err, amax)
