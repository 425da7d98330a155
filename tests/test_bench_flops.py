"""The FLOPs that bench.py's rooflines credit to the octant kernels are the ones they do (sym.cuh):
class members padded to tiles of 8 or steps of 4, over the nq / 8 octant directions."""
import importlib.util
import os

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_spec = importlib.util.spec_from_file_location("bench", os.path.join(REPO, "bench.py"))
bench = importlib.util.module_from_spec(_spec)
_spec.loader.exec_module(bench)


@pytest.mark.parametrize("N", range(8))
def test_octant_classes_hold_every_harmonic(N):
    n = bench._octant_classes(N)
    assert sum(n) == (N + 1) ** 2
    # odd under all three flips: l odd, m < 0 even -- first (3, -2)
    assert (n[7] > 0) == (N >= 3)


def test_m6_counts_are_the_kernels():
    """M_6, classes of 10, 6 (six times) and 3 members: per block of 8 octant directions and 8 cells a
    probe expands with 3 + 6 * 2 + 1 = 16 DMMAs and projects onto 2 + 7 = 9 tiles, twice; a pass onto
    24. A DMMA has 512 FLOPs, a block 64 pairs of cell and octant direction."""
    nm, nq = 49, 1568
    other = nq / 8 * (24 + 8 + 8 + 24)
    assert bench.octant_pass_flops(nm, nq, 6) - other == nq / 8 * (16 + 2 * 9) * 512 / 64
    assert bench.octant_pass_flops(nm, nq, 12) - other == nq / 8 * (16 + 2 * 24) * 512 / 64
    assert bench.octant_stencil_flops(nm, nq) == nq * 60 + nq / 8 * (24 + 9 * 16)


@pytest.mark.parametrize("N", [2, 4, 6, 7])
def test_octant_counts_are_below_the_full_ones(N):
    nm, nq = (N + 1) ** 2, 2 * (2 * (N + 3)) ** 2
    assert bench.octant_stencil_flops(nm, nq) < (2 * nm + 60) * nq
    assert bench.octant_pass_flops(nm, nq, N) < 4 * nm * nq + nq
