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


# scenes large enough for the stress update of one thread per particle, in the
# instantiation of each material type (smaller ones, as in the parity cases,
# share a particle's gather among three warps)
LARGE = {
    "elastic": lambda d: d.generic_block("1 elas 1000 1e7 0.3", counts=(24, 22, 20)),
    "plastic_gimp": lambda d: d.generic_block("1 pla1 1000 1e7 0.3 2e4", counts=(24, 22, 20), shape="gimp", scheme="musl"),
    "bar_johnson_cook": lambda d: d.taylor_bar(dp=4e-4),
    "dam_null_bspline": lambda d: d.dam_break(dp=0.1, h=0.2),
    "slope_drucker_prager_gimp": lambda d: d.soil_slope(dp=0.4, width=3.2),
    "beam_neo_hookean_sgmp": lambda d: d.soft_beam(dp=0.1, length=10.0),
}


@pytest.mark.parametrize("name", sorted(LARGE))
def test_large_scene(gpu_mod, oracle_mod, name):
    from mpm3d_gb300 import decks
    text = LARGE[name](decks)
    g, o = run_pair(gpu_mod, oracle_mod, text, STEPS, "fp64", "project")
    assert g.download("VXp").shape[-1] > 9728
    check_strict(g, o, name, STEPS)
