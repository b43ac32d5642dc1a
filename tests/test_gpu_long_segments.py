"""Keys of the batched engine's re-sort that hold more particles than a block
sorts in shared memory (8192): the particles outside a scene's grid all share
one. Ordering them is linear work, so that a wait beside it stays short, and
gives the stable order whether they lie together in the deck or strewn over it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ["Xp", "VXp", "SM", "ie"]
STEPS = 2
# about 8 ms: the other phases of these sorts take under 1 ms, a bitonic
# network over the long key in global memory 17 ms (216 k particles) to 94 ms (1 M)
POLLS = 20000


def _block(n, spans):
    from mpm3d_gb300 import decks
    return decks.generic_block("1 elas 1000 1e6 0.3", counts=n, shape="gimp", gravity=None, velocity=(0.3, 0.2, 0.1),
                               dtscale=0.3, fixed="0 0 0 0 0 0", extra=spans)


def _check(text, polls):
    from mpm3d_gb300 import Batch, Deck, MpmStep, decks
    d = Deck.parse(text)
    x = d.particles()["Xp"]
    other = Deck.parse(decks.soil_slope(dp=0.5, width=2.0))
    runs = []
    for lead in (False, True):
        with Batch() as b:
            b.set_option("sort_polls", polls)
            if lead:
                b.add(other, steps=STEPS)
            s = b.add(d, steps=STEPS)
            b.run(STEPS)
            b.sync()
            runs.append(([b.download(s, f) for f in FIELDS], b.scalars(s)))
    (a, sa), (c, sc) = runs
    for f, u, v in zip(FIELDS, a, c):
        np.testing.assert_array_equal(u, v, err_msg=f)
    assert sa == sc  # the energies are sums in the particles' order
    r = MpmStep(d, "fp64")
    r.run(STEPS)
    for f, u in zip(FIELDS[:2], a):
        w = r.download(f)
        assert np.max(np.abs(u - w)) <= 1e-6 * np.max(np.abs(w)), f
    return x


@pytest.mark.parametrize("n", [22, 60, 100])
def test_most_outside(built, n):
    """All but a corner of 12^3 particles of n^3 outside the grid."""
    x = _check(_block((n, n, n), ("spx -2 6", "spy -2 6", "spz -2 7")), POLLS)
    out = np.any(x > np.array([[6], [6], [7]]), axis=0)
    assert out.sum() > 8192


def test_strewn_outside(built):
    """Every hundredth particle of the deck outside: 10 000 among a million (a
    network of 10 000 is short)."""
    x = _check(_block((100, 100, 100), ("spx -1.5 49.5", "spy -2 52", "spz -1 56")), POLLS)
    out = np.flatnonzero(x[0] > 49.5)
    assert len(out) == 10000 and out[-1] - out[0] > 64 * len(out)
