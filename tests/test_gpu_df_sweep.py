"""The dataflow sweep on triangles of about as many rows as its ring has slots.

A ring slot is overwritten once the writer warp has reported that its row is
in global memory; the reports may lag by 64 rows, so that a ring of 256 slots
with a reach of up to 56 rows always moves on. Plates of 256 to 533 rows
(just as many rows as slots, a few more, and two rounds of the ring), and 1,024
rows, each against the oracle's triangular solves to 1e-12 of max |z| (the gate
of the other sweeps).
"""
import numpy as np
import pytest

from gpu_fem_b200 import mesh as M

pytestmark = pytest.mark.gpu

CASES = [(15, 15, 3), (16, 15, 3), (16, 16, 3), (19, 15, 1), (40, 12, 3), (31, 31, 0)]


@pytest.mark.parametrize("nx,ny,fill", CASES)
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_dataflow_sweep_around_its_ring(nx, ny, fill, precision):
    import torch
    from gpu_fem_b200.assembler import ElementAssembler, ILUk_Preconditioner, createBsrMat
    from oracle import pyoracle as po
    m = M.plate(nx, ny, 1.0, ny / nx, lambda x, y: 0.006 + 0 * x, "all_edges",
                lambda q: 1e3 + 0 * q[:, 0])
    A = ElementAssembler.from_mesh(m, ordering="natural")
    K = createBsrMat(A)
    A.add_jacobian(None, K, fuse_bcs=True)
    P = ILUk_Preconditioner(A, fill, precision, sweep="dataflow")
    P.factor(K)
    assert P.sweeps()["L"] == "dataflow"
    rowp, cols, lu = P.get()
    used = lu.astype(np.float32).astype(np.float64) if precision == "fp32" else lu
    for seed in (1, 2):
        r = np.random.default_rng(seed).standard_normal(m.num_dof)
        z = torch.full((m.num_dof,), float("nan"), dtype=torch.float64, device="cuda")
        P.apply(torch.tensor(r, device="cuda"), z)
        assert P.status() == 0
        ref = po.ilu_apply_dinv(rowp, cols, used, r)
        assert np.abs(z.cpu().numpy() - ref).max() <= 1e-12 * np.abs(ref).max()
