"""A wait inside the batched engine's re-sort that runs out (a limit of one poll
makes it) reaches the caller from whatever he calls next, and the batch can be
used again once its scenes are gone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TIMEOUT = 8  # MPM_ERR_TIMEOUT


def _deck():
    from mpm3d_gb300 import Deck, decks
    return Deck.parse(decks.soil_slope(dp=0.4, width=2.0))  # some 250 blocks


def _stalled(graph=True):
    from mpm3d_gb300 import Batch
    b = Batch()
    b.set_option("sort_polls", 1)
    s = b.add(_deck(), steps=40)
    b.commit()
    b.run(3, graph=graph)  # (the first step of a scene sorts it)
    return b, s


CALLS = {
    "sync": lambda b, s: b.sync(),
    "scalars": lambda b, s: b.scalars(s),
    "download": lambda b, s: b.download(s, "Xp"),
    "run_then_scalars": lambda b, s: (b.run(1), b.scalars(s)),
    "run_loop": lambda b, s: b.run_loop(4),
    "time_steps": lambda b, s: b.time_steps(2),
    "commit_beside_another": lambda b, s: (b.add(_deck(), steps=4), b.commit()),
    "download_beside_another": lambda b, s: (b.add(_deck(), steps=4), b.download(s, "Xp")),
}


@pytest.mark.parametrize("call", sorted(CALLS))
@pytest.mark.parametrize("graph", [True, False])
def test_reported(built, call, graph):
    from mpm3d_gb300 import MpmError
    b, s = _stalled(graph)
    with b:
        for _ in range(2):  # (it stays reported)
            with pytest.raises(MpmError) as e:
                CALLS[call](b, s)
            assert e.value.code == TIMEOUT, e.value


def test_first_call_of_a_loop(built):
    from mpm3d_gb300 import Batch, MpmError
    with Batch() as b:
        b.set_option("sort_polls", 1)
        b.add(_deck(), steps=40)
        with pytest.raises(MpmError) as e:
            b.run_loop(8)
        assert e.value.code == TIMEOUT


def test_batch_goes_on_without_its_scenes(built):
    from mpm3d_gb300 import MpmError, MpmStep
    b, s = _stalled()
    with b:
        with pytest.raises(MpmError):
            b.sync()
        b.remove(s)
        b.set_option("sort_polls", 0)
        t = b.add(_deck(), steps=5)
        b.run(5)
        b.sync()
        m = MpmStep(_deck(), "mixed")
        m.run(5)
        for f in ("Xp", "VXp", "SM"):
            np.testing.assert_array_equal(b.download(t, f), m.download(f), err_msg=f)
