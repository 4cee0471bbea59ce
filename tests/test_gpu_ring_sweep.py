"""The default triangular sweep against the oracle's triangular solves.

P.apply with sweep="auto" on the GPU's own factor values, checked entry by
entry to 1e-12 of max |z| (the gate of the other sweeps: products of at most
a few hundred blocks accumulate in FP64 on both sides). Cases sit where the
layout changes: rows of up to 16 blocks (one pass), of 17 to 32 and more
(shared by warps, or several passes of one warp where every warp has a row),
levels with more rows than warps, one CTA and clusters of two and four,
complete factors, and a numbering whose dependency reach does not fit the
shared-memory ring (solved by the chunked sweep).
"""
import numpy as np
import pytest

from gpu_fem_b200 import mesh as M

pytestmark = pytest.mark.gpu

FULL = 0x7FFFFFFF
CASES = {
    "one_element": (1, 1, 2, "natural"), "ilu0_strip": (2, 1, 0, "natural"),
    "ilu0_wide": (90, 40, 0, "rcm"), "short_rows": (40, 16, 6, "natural"),
    "shared_rows": (17, 16, 8, "natural"), "three_passes": (48, 40, 16, "natural"),
    "full": (40, 20, FULL, "natural"), "long_full": (60, 45, FULL, "natural"),
    "many_rows": (300, 40, 2, "natural"), "cluster": (200, 60, 8, "natural"),
    "rcm": (61, 37, 10, "rcm"), "no_ring": (90, 90, 0, "shuffled"),
}


def _factored(case, precision):
    import torch
    from gpu_fem_b200.assembler import ElementAssembler, ILUk_Preconditioner, createBsrMat
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
    P = ILUk_Preconditioner(A, fill, precision)
    P.factor(K)
    torch.cuda.synchronize()
    return m, A, K, P


@pytest.mark.parametrize("case", list(CASES))
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_default_sweep_matches_oracle(case, precision):
    import torch
    from oracle import pyoracle as po
    m, A, K, P = _factored(case, precision)
    assert P.sweeps()["L"] == "level"
    rowp, cols, lu = P.get()
    used = lu.astype(np.float32).astype(np.float64) if precision == "fp32" else lu
    for seed in (1, 2):  # the second apply meets the first one's leftovers
        r = np.random.default_rng(seed).standard_normal(m.num_dof)
        z = torch.full((m.num_dof,), float("nan"), dtype=torch.float64, device="cuda")
        P.apply(torch.tensor(r, device="cuda"), z)
        assert P.status() == 0
        ref = po.ilu_apply_dinv(rowp, cols, used, r)
        assert np.abs(z.cpu().numpy() - ref).max() <= 1e-12 * np.abs(ref).max()


def test_default_sweep_timeout_is_reported():
    """A cluster whose CTA of rank 1 sends no results: the others' bounded
    waits run out, the status reports it, and the next apply is correct."""
    import torch
    from gpu_fem_b200 import _lib as L
    m, A, K, P = _factored("cluster", "fp64")
    assert P.layout()["nsplit_L"] == 2
    r = torch.tensor(np.random.default_rng(3).standard_normal(m.num_dof), device="cuda")
    z0, z1 = torch.zeros_like(r), torch.zeros_like(r)
    P.apply(r, z0)
    assert P.status() == L.GF_OK
    torch.cuda.synchronize()
    try:
        L.check(L.lib().gf_test_set_waits(200_000, 1), "set_waits")
        P.apply(r, z1)
        assert P.status() == L.GF_TIMEOUT
    finally:
        L.check(L.lib().gf_test_set_waits(0, 0), "restore waits")
    P.apply(r, z1)
    assert P.status() == L.GF_OK
    assert torch.equal(z0, z1)


@pytest.mark.parametrize("tail", [3, 60])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_default_sweep_levels_of_one_row(tail, precision):
    """A plate wide enough for a cluster with a strip one element wide at its
    far corner: the lower sweep ends and the upper one begins with long runs
    of levels in which only one CTA has a row. Same gate as above."""
    import torch
    from gpu_fem_b200.assembler import ElementAssembler, ILUk_Preconditioner, createBsrMat
    from oracle import pyoracle as po
    nx, ny = 200, 60
    m = M.plate(nx, ny + tail, 1.0, 0.3, lambda x, y: 0.006 + 0 * x, "x0",
                lambda q: 1e3 + 0 * q[:, 0])
    e = np.arange(m.conn.shape[0])
    keep = (e // nx < ny) | (e % nx == nx - 1)
    m.conn, m.thick = m.conn[keep], m.thick[keep]
    nodes = np.unique(m.conn)
    new = np.full(m.num_nodes, -1)
    new[nodes] = np.arange(len(nodes))
    m.conn, m.xpts = new[m.conn].astype(np.int32), m.xpts[nodes]
    bcs = m.bcs[new[m.bcs // 6] >= 0]
    m.bcs = (6 * new[bcs // 6] + bcs % 6).astype(np.int32)
    A = ElementAssembler.from_mesh(m, ordering="natural")
    K = createBsrMat(A)
    A.add_jacobian(None, K, fuse_bcs=True)
    P = ILUk_Preconditioner(A, 8, precision)
    P.factor(K)
    assert P.layout()["nsplit_L"] == 2 and P.layout()["nsplit_U"] == 2
    rowp, cols, lu = P.get()
    used = lu.astype(np.float32).astype(np.float64) if precision == "fp32" else lu
    for seed in range(3):
        r = np.random.default_rng(seed).standard_normal(m.num_dof)
        z = torch.full((m.num_dof,), float("nan"), dtype=torch.float64, device="cuda")
        P.apply(torch.tensor(r, device="cuda"), z)
        assert P.status() == 0
        ref = po.ilu_apply_dinv(rowp, cols, used, r)
        assert np.abs(z.cpu().numpy() - ref).max() <= 1e-12 * np.abs(ref).max()
