"""Batches of many scenes of both families of node kernels (SGMP and the others),
added in any order, joined and left on the way, of more scenes than the block
that starts a step has threads, each moving on its own so that it is re-sorted
in steps of its own: every scene ends as it does alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ["Xp", "VXp", "SM", "SD", "PXg"]


def _deck(shape, n, v):
    from mpm3d_gb300 import Deck, decks
    return Deck.parse(decks.generic_block("1 elas 1000 1e5 0.3", counts=(n, n, n), shape=shape, scheme="musl", gravity=None,
                                          velocity=v, dtscale=0.4, fixed="0 0 0 0 0 0",
                                          extra=("spx -8 16", "spy -8 16", "spz -8 16")))


def _alone(d, steps):
    from mpm3d_gb300 import MpmStep
    m = MpmStep(d, "mixed")
    m.run(steps)
    return [m.download(f) for f in FIELDS]


def _same(b, s, want, what):
    for f, w in zip(FIELDS, want):
        np.testing.assert_array_equal(b.download(s, f), w, err_msg=f"{what} {f}")


@pytest.mark.parametrize("order", [("sgmp", "gimp", "sgmp", None), (None, "bimp", "sgmp"), ("sgmp", "sgmp"), ("gimp", "sgmp")])
def test_families_in_any_order(built, order):
    from mpm3d_gb300 import Batch
    rng = np.random.default_rng(5)
    ds = [_deck(s, int(rng.integers(2, 9)), tuple(rng.uniform(-2, 2, 3))) for s in order]
    late = _deck("gimp", 5, (1.0, -1.5, 0.5))
    with Batch() as b:
        ids = [b.add(d, steps=30) for d in ds]
        b.run(10)
        j = b.add(late, steps=15)
        b.run(10)
        b.remove(ids[0])
        b.run(20)
        b.sync()
        for k in range(1, len(ds)):
            _same(b, ids[k], _alone(ds[k], 30), f"{order} {k}")
        _same(b, j, _alone(late, 15), f"{order} late")


@pytest.mark.parametrize("n", [1, 255, 256, 257, 600])
def test_number_of_scenes(built, n):
    from mpm3d_gb300 import Batch
    rng = np.random.default_rng(n)
    shapes = [None, "gimp", "bimp", "sgmp"]
    ds = [_deck(shapes[k], k + 3, tuple(rng.uniform(-2, 2, 3))) for k in range(4)] + \
         [_deck(shapes[k % 4], 4, tuple(rng.uniform(-3, 3, 3))) for k in range(9)]
    with Batch() as b:
        pick = [int(rng.integers(len(ds))) for _ in range(n)]
        steps = [int(rng.integers(5, 30)) for _ in range(n)]
        ids = [b.add(ds[p], steps=s) for p, s in zip(pick, steps)]
        b.run(30)
        b.sync()
        for k in sorted({0, n // 3, n // 2, n - 1} | {int(x) for x in rng.integers(n, size=6)}):
            assert b.scalars(ids[k])["istep"] == steps[k]
            _same(b, ids[k], _alone(ds[pick[k]], steps[k]), f"scene {k} of {n}")
