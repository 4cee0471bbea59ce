"""Creating an assembler spends its time on the mesh, not on scatter tables.

The records of the blocks and nodes that each chunk of elements contributes to
follow from the elemIndMap with a few operations per entry, far less than the
ordering and the colouring of the mesh on the host: their share of the setup
of a 400x200 plate is at most a quarter (the best of five setups each: a busy
host can only lengthen them).
"""
import pytest

from gpu_fem_b200 import mesh as M

pytestmark = pytest.mark.gpu


def test_chunk_records_are_a_small_part_of_the_setup():
    from gpu_fem_b200.assembler import ElementAssembler
    m = M.plate(400, 200, 1.0, 0.5, lambda x, y: 0.006 + 0 * x, "all_edges",
                lambda q: 1e3 + 0 * q[:, 0])
    times = [ElementAssembler.from_mesh(m).setup_times() for _ in range(5)]
    records, setup = (min(t[k] for t in times) for k in ("records_ms", "setup_ms"))
    assert 0.0 < records <= 0.25 * setup, times
