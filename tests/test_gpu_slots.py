"""Influence slots of the FP64 forms against the oracle, bit for bit: particles
in every part of their cells (cpGIMP: 8, 12, 18 and 27 slots, in lists whose
lengths are no multiple of a warp), and particles in the grid's first and last
cells, whose offsets leave the grid or cross the end of a row."""
import pytest

from gpu_cases import check_strict, run_pair

pytestmark = pytest.mark.gpu

STEPS = 4


@pytest.mark.parametrize("shape", [None, "gimp", "bimp", "sgmp"])
@pytest.mark.parametrize("counts", [(1, 1, 1), (5, 4, 7), (11, 13, 6)])
@pytest.mark.parametrize("edge", [False, True])
def test_slots(gpu_mod, oracle_mod, shape, counts, edge):
    from mpm3d_gb300 import decks
    dp = 0.37
    if edge:  # the block fills the grid up to a part of a cell
        span = [(0, int(counts[0] * dp) + 1), (0, int(counts[1] * dp) + 1), (0, int((counts[2] + 2) * dp) + 1)]
    else:
        span = [(-3, 9), (-3, 9), (-3, 9)]
    text = decks.generic_block("1 elas 1000 1e5 0.3", dp=dp, counts=counts, shape=shape, scheme="musl",
                               velocity=(0.3, -0.1, 0.2) if not edge else (0.0, 0.0, 0.0), fixed="2 2 2 2 2 2",
                               extra=("dcel 1.0",) + tuple("sp%s %d %d" % (a, *s) for a, s in zip("xyz", span)))
    g, o = run_pair(gpu_mod, oracle_mod, text, STEPS, "fp64", "project")
    check_strict(g, o, f"{shape} {counts} {edge}", STEPS)
