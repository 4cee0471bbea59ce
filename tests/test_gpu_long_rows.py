"""Preconditioners with long rows: what is refused, and what the setup costs.

A factor whose longest row the chunked level sweep cannot stage in shared
memory is refused with the default sweep too, whichever kernel would solve it:
complete factors of natural-order plates with rows on both sides of the limit
are accepted and refused alike by "auto" and "level". (Two stages of 296 bytes
a block, FP32 152, and 96 bytes a block for the gathered x have to fit 188,320
bytes: 273 blocks in FP64, 470 in FP32; U has nx + 3 in a row.) The default
sweep's setup only counts those chunks; it lays out one kind of stream. On a
plate of 140 elements in width the chunked streams take most of a setup, so
that the one with the default sweep takes at most half as long as the one with
"level" (the best of three each, without the ILU pattern).
"""
import numpy as np
import pytest

from gpu_fem_b200 import mesh as M

pytestmark = pytest.mark.gpu

FULL = 0x7FFFFFFF


def _assembler(nx, ny):
    from gpu_fem_b200.assembler import ElementAssembler
    m = M.plate(nx, ny, 1.0, ny / nx, lambda x, y: 0.006 + 0 * x, "all_edges",
                lambda q: 1e3 + 0 * q[:, 0])
    return ElementAssembler.from_mesh(m, ordering="natural")


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_auto_refuses_what_level_refuses(precision):
    from gpu_fem_b200 import _lib as L
    from gpu_fem_b200.assembler import ILUk_Preconditioner
    seen = set()
    limit = 273 if precision == "fp64" else 470
    for nx in range(limit - 11, limit + 6, 2):
        A = _assembler(nx, 3)
        accepted = []
        for sweep in ("auto", "level"):
            try:
                ILUk_Preconditioner(A, FULL, precision, sweep=sweep)
                accepted.append(True)
            except L.GpuFemError as e:
                assert e.status == L.GF_INVALID_ARG and "rows too long" in str(e)
                accepted.append(False)
        assert accepted[0] == accepted[1], nx
        seen.add(accepted[0])
    assert seen == {True, False}


def test_auto_lays_out_one_stream():
    from gpu_fem_b200.assembler import ILUk_Preconditioner
    A = _assembler(140, 30)
    best = {}
    for sweep in ("auto", "level"):
        t = []
        for _ in range(3):
            P = ILUk_Preconditioner(A, FULL, "fp64", sweep=sweep)
            n = np.diff(P.get()[0])
            assert n.max() > 2 * 136
            i = P.setup_info()
            t.append(i["setup_ms"] - i["symbolic_ms"])
        best[sweep] = min(t)
    assert best["auto"] <= 0.5 * best["level"], best
