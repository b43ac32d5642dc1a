"""The FP64 forms in grids of many more nodes than the particles reach, which
finish the empty nodes apart from the others (fewer blocks than groups of
nodes) and look for segments to order many nodes at a time (from 65536 nodes
on): bit-identical to the oracle, with segments of every length among them."""
import numpy as np
import pytest

from gpu_cases import check_strict, run_pair

pytestmark = pytest.mark.gpu

STEPS = 3


def _deck(shape, scheme, n, cells, dp):
    from mpm3d_gb300 import decks
    # off the middle, so that empty nodes lie before and behind the others
    lo, hi = -2 - cells // 3, cells - 2 - cells // 3
    return decks.generic_block("1 elas 1000 1e5 0.3", dp=dp, counts=(n, n, n), shape=shape, scheme=scheme,
                               velocity=(1.7, 0.9, -2.3), fixed="0 0 0 0 0 0",
                               extra=("dcel 1.0", f"spx {lo} {hi}", f"spy {lo} {hi}", f"spz {lo} {hi}"))


@pytest.mark.parametrize("shape", [None, "gimp", "bimp", "sgmp"])
@pytest.mark.parametrize("scheme", ["usf", "usl", "musl"])
@pytest.mark.parametrize("n,cells,dp", [(1, 20, 0.5), (5, 45, 0.5), (7, 41, 0.15)])
def test_sparse(gpu_mod, oracle_mod, shape, scheme, n, cells, dp):
    g, o = run_pair(gpu_mod, oracle_mod, _deck(shape, scheme, n, cells, dp), STEPS, "fp64", "project")
    check_strict(g, o, f"{shape} {scheme} {n} {cells}", STEPS)
    assert g.scalars()["active_nodes"] == np.count_nonzero(o.download("Mg") > 0)


@pytest.mark.parametrize("shape", [None, "sgmp"])
def test_very_sparse(gpu_mod, oracle_mod, shape):
    """A million nodes: sixteen at a time."""
    g, o = run_pair(gpu_mod, oracle_mod, _deck(shape, "musl", 6, 100, 0.25), 2, "fp64", "project")
    check_strict(g, o, f"{shape}", 2)
