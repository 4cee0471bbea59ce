"""Assembly at the edges of its element chunks.

Chunks hold up to eight elements: meshes of 1 to 35 elements end in every
remainder, and fans of quads around one node give that node's diagonal block
up to eight contributions of one chunk, and more over several chunks. K and R
against the oracle within 1e-12 / 1e-11 of max |K| / |R| (the gates of the
other assembly tests); the residual kernel, which shares no strain code with
the Jacobian, against R = K u within 1e-12 with a thickness offset and a
reference axis too (sums of at most a few hundred FP64 products each).
"""
import numpy as np
import pytest

from gpu_fem_b200 import mesh as M

pytestmark = pytest.mark.gpu


def _fan(n):
    """n quads (centre, p_i, p_{i+1}, q_i) around node 0, bent out of plane."""
    a = 2 * np.pi * np.arange(n) / n
    p = np.stack([np.cos(a), np.sin(a), 0.2 * np.cos(2 * a)], 1)
    q = 1.6 * np.stack([np.cos(a + np.pi / n), np.sin(a + np.pi / n), 0.1 + 0 * a], 1)
    x = np.concatenate([np.zeros((1, 3)), p, q])
    i = np.arange(n)
    conn = np.stack([0 * i, 1 + i, 1 + (i + 1) % n, 1 + n + i], 1).astype(np.int32)
    return M.ShellMesh(conn, x, np.linspace(0.004, 0.009, n), np.array([6, 8, 11], np.int32),
                       np.zeros(6 * len(x)), name=f"fan_{n}")


def _panel(nx, ny):
    m = M.plate(nx, ny, 1.0, 0.7, lambda x, y: 0.004 + 0.003 * x, "x0", lambda q: 1e3 + 0 * q[:, 0],
                jitter=0.1)
    m.xpts[:, 2] = 0.1 * np.sin(2 * m.xpts[:, 0]) * np.cos(m.xpts[:, 1])
    return m


MESHES = {"fan3": lambda: _fan(3), "fan8": lambda: _fan(8), "fan9": lambda: _fan(9),
          "fan20": lambda: _fan(20), "1x1": lambda: _panel(1, 1), "3x1": lambda: _panel(3, 1),
          "3x3": lambda: _panel(3, 3), "5x7": lambda: _panel(5, 7)}


@pytest.mark.parametrize("name", list(MESHES))
def test_chunk_edges_match_oracle(oracle, name):
    import torch
    from gpu_fem_b200.assembler import ElementAssembler, createBsrMat
    m = MESHES[name]()
    u = np.random.default_rng(2).standard_normal(m.num_dof) * 1e-3
    A = ElementAssembler.from_mesh(m)
    A.set_variables(A.createVarsVec(u))
    K, K2, R, R2 = createBsrMat(A), createBsrMat(A), A.createVarsVec(), A.createVarsVec()
    A.add_jacobian(R, K)
    A.add_jacobian(R2, K2, fuse_bcs=True)
    torch.cuda.synchronize()
    rowp, cols, vals, r, perm = oracle.assemble_jacobian(m, u)
    assert np.abs(K.values_host() - vals).max() <= 1e-12 * np.abs(vals).max()
    assert np.abs(R.t.cpu().numpy() - r).max() <= 1e-11 * np.abs(r).max()
    oracle.apply_bcs_mat(rowp, cols, vals, perm, m.bcs)
    assert np.abs(K2.values_host() - vals).max() <= 1e-12 * np.abs(vals).max()
    r[m.bcs] = 0.0
    assert np.abs(R2.t.cpu().numpy() - r).max() <= 1e-11 * np.abs(r).max()
    # added to what is there
    A.add_jacobian(R2, K2, fuse_bcs=True, add=True)
    A.add_residual(R, add=True)
    torch.cuda.synchronize()
    assert np.abs(K2.values_host() - 2 * vals).max() <= 2e-12 * np.abs(vals).max()
    assert np.abs(R2.t.cpu().numpy() - 2 * r).max() <= 2e-11 * np.abs(r).max()


@pytest.mark.parametrize("name", ["fan9", "5x7"])
@pytest.mark.parametrize("offset,axis", [(0.0, None), (0.3, (1.0, 0.3, 0.2))])
def test_residual_and_energy_agree_with_jacobian(name, offset, axis):
    import torch
    from gpu_fem_b200.assembler import ElementAssembler, createBsrMat
    m = MESHES[name]()
    u = np.random.default_rng(4).standard_normal(m.num_dof) * 1e-3
    A = ElementAssembler.from_mesh(m, tOffset=offset, ref_axis=axis)
    A.set_variables(A.createVarsVec(u))
    K, R, R2 = createBsrMat(A), A.createVarsVec(), A.createVarsVec()
    A.add_jacobian(R, K)
    A.add_residual(R2)
    y = torch.zeros(m.num_dof, dtype=torch.float64, device="cuda")
    K.spmv(torch.tensor(u, device="cuda"), y)
    torch.cuda.synchronize()
    r, r2, y = R.t.cpu().numpy(), R2.t.cpu().numpy(), y.cpu().numpy()
    assert np.abs(r - y).max() <= 1e-12 * np.abs(y).max()
    assert np.abs(r2 - y).max() <= 1e-12 * np.abs(y).max()
    e = 0.5 * float(u @ y)
    assert abs(A.add_energy() - e) <= 1e-12 * abs(e)
