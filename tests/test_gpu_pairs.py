"""The node-sorted pair list of the FP64 forms: nodes whose segments are as
long as each way of ordering them takes (32, 64, 128 and 256 pairs by one
warp, longer ones by one block, in shared memory or beyond it) are summed in
the reference's order, so the strict form stays bit-identical to the oracle."""
import pytest

from gpu_cases import check_strict, run_pair

pytestmark = pytest.mark.gpu

STEPS = 3


@pytest.mark.parametrize("shape,n", [(None, 3), (None, 4), ("sgmp", 4), (None, 5), ("bimp", 5), ("sgmp", 6), (None, 6),
                                     ("gimp", 7), (None, 21), ("sgmp", 21)])
def test_segment_lengths(gpu_mod, oracle_mod, shape, n):
    """A cube of n^3 particles about as wide as one cell: up to n^3 pairs at a
    node (more by the wider shapes)."""
    from mpm3d_gb300 import decks
    text = decks.generic_block("1 elas 1000 1e5 0.3", dp=1.0 / n, counts=(n, n, n), shape=shape, scheme="musl",
                               velocity=(1.7, 0.9, -2.3), fixed="0 0 0 0 0 0",
                               extra=("dcel 1.0", "spx -3 4", "spy -3 4", "spz -2 5"))
    g, o = run_pair(gpu_mod, oracle_mod, text, STEPS, "fp64", "project")
    check_strict(g, o, f"{shape} {n}", STEPS)
