"""Re-sorting of the batched engine's particles: a scene that crosses many
cells is re-sorted on its own particles' disorder only, so its results are the
same alone, beside scenes that keep their order, and however its run is split;
and they stay within the mixed form's bound of FP64."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ["Xp", "VXp", "SM", "SD", "PXg"]
STEPS = 60


def _moving(shape, n):
    """An elastic block of n^3 particles (h = 1 m) flying diagonally at up to
    a third of a cell per step: particles leave their keys at rates from none
    to most of them between steps."""
    from mpm3d_gb300 import decks
    return decks.generic_block("1 elas 1000 1e5 0.3", counts=(n, n, n), shape=shape, scheme="musl", gravity=None,
                               velocity=(1.7, 0.9, 2.3), dtscale=0.4, fixed="0 0 0 0 0 0",
                               extra=("spx -20 60", "spy -20 60", "spz 0 90"))


@pytest.mark.parametrize("shape,n", [(None, 3), (None, 17), ("gimp", 10), ("gimp", 21), ("bimp", 13), ("sgmp", 11)])
def test_resorted_scene_identity(built, shape, n):
    from mpm3d_gb300 import Batch, Deck, MpmStep, decks
    d = Deck.parse(_moving(shape, n))
    rest = Deck.parse(decks.soil_slope(dp=0.5, width=2.0))
    m = MpmStep(d, "mixed")
    m.run(STEPS)
    want = {f: m.download(f) for f in FIELDS}
    x0 = d.particles()["Xp"]
    assert np.min(np.abs(want["Xp"] - x0).max(axis=1)) > 1.0  # every direction crossed a cell
    with Batch() as bt:
        bt.add(rest, steps=STEPS)
        a = bt.add(d, steps=STEPS)
        bt.add(rest, steps=STEPS)
        for k in (1, 7, 20, 32):
            bt.run(k, graph=k != 7)
        bt.sync()
        for f in FIELDS:
            np.testing.assert_array_equal(bt.download(a, f), want[f], err_msg=f"{shape} {n} {f}")
    r = MpmStep(d, "fp64")
    r.run(STEPS)
    for f in FIELDS:
        b = r.download(f)
        s = np.max(np.abs(b))
        # a block in uniform flight carries rounding-size stresses only: they
        # are compared on the scale of E, 1e5 Pa
        scale = 1e5 if f in ("SM", "SD") else s
        assert np.max(np.abs(want[f] - b)) <= 1e-5 * scale, f"{shape} {n} {f}"


@pytest.mark.parametrize("shape", [None, "gimp", "bimp", "sgmp"])
def test_resorted_restart(built, tmp_path, shape):
    """A restart between two re-sorts continues bit-identically."""
    from mpm3d_gb300 import Deck, MpmStep
    d = Deck.parse(_moving(shape, 9))
    a = MpmStep(d, "mixed")
    a.run(33)
    a.save(str(tmp_path / "r"))
    a.run(27)
    b = MpmStep(d, "mixed")
    b.load(str(tmp_path / "r"))
    b.run(27)
    for f in FIELDS:
        np.testing.assert_array_equal(a.download(f), b.download(f), err_msg=f"{shape} {f}")


@pytest.mark.parametrize("thick", [1.0, 1.25, 2.25])
def test_sgmp_every_shear(built, thick):
    """Every stress component of the SGMP transfers: a neo-Hookean cantilever
    (4, 5 and 9 layers across, a mostly empty grid, no side walls) under an
    oblique body force bends about both axes and shears in every plane; the
    mixed form stays within its bound of FP64 in each field, the node forces
    included."""
    from mpm3d_gb300 import Deck, MpmStep, decks
    text = decks.soft_beam(thick=thick)
    span = "spy 0 %.9g" % thick
    assert span in text and "fixe 1 0 2 2 0 0" in text and "grav 1 0 0 -9.8" in text
    text = text.replace(span, "spy -2 4.5").replace("fixe 1 0 2 2 0 0", "fixe 1 0 0 0 0 0")
    text = "\n".join("grav 1 4 7 -9" if ln.startswith("grav") else ln for ln in text.splitlines()) + "\n"
    d = Deck.parse(text)
    a, b = MpmStep(d, "fp64"), MpmStep(d, "mixed")
    a.run(60)
    b.run(60)
    for f in FIELDS + ["FXg"]:
        x, y = a.download(f), b.download(f)
        err = np.max(np.abs(x - y)) / np.max(np.abs(x))
        assert err <= 1e-5, f"thick {thick} {f}: {err:.3g}"
    sd = a.download("SD")
    assert np.all(np.max(np.abs(sd[3:]), axis=1) > 1e-3 * np.max(np.abs(sd)))  # every shear takes part
