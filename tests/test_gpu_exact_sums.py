"""The mixed form's particle -> node sums are rounded within one key's particles
only: across keys they are added in fixed point. Every weight, mass and
velocity here is a short binary fraction, so that a key's FP32 sum is exact,
while the masses of neighbouring columns differ by 2^9, so that the sum of two
keys does not fit FP32's 24 bits. The node sums then equal the FP64 form's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NX, NY = 16, 3


def _text(shape, scheme, gravity):
    """8 particles about the centre of every unit cell (linear) or about every
    node (GIMP and SGMP, whose keys are the nearest node and the dual cell), in
    key order; column i along x has masses of 12 bits times 2^(9 (i mod 3))."""
    from mpm3d_gb300.decks import DeckWriter, _grid_lines
    w = DeckWriter("sums")
    w.kw("nmat 1")
    w.head += _grid_lines(((-3, NX + 4), (-3, NY + 4), (-3, NY + 4)), 1.0)
    # (a material so soft that its forces are below the last FP32 bit of the sums)
    for line in ("dtsc 1e-6", "endt 100.0", f"{scheme} on") + ((shape,) if shape else ()) + (
            "fixe 0 0 0 0 0 0", "mate", "1 elas 1000 1e-6 0.3"):
        w.kw(line)
    at = 0.0 if shape else 0.5
    q = np.array([(x, y, z) for z in (-0.25, 0.25) for y in (-0.25, 0.25) for x in (-0.25, 0.25)])
    xyz, mass = [], []
    for k in range(NY):
        for j in range(NY):
            for i in range(NX):
                xyz.append(q + (i + 1 + at, j + 1 + at, k + 1 + at))
                mass.append(np.full(8, (2049 + 2 * i) * 2.0 ** (9 * (i % 3))))
    w.points(1, np.concatenate(mass), np.concatenate(xyz))
    w.tail += ["velo", "body 1 0.5 0.25 -0.75", "endv"]
    if gravity:
        w.tail += ["load", "grav 1 2 4 -8", "endl"]
    return w.text()


def _deck(*a):
    from mpm3d_gb300 import Deck
    return Deck.parse(_text(*a))


@pytest.mark.parametrize("shape", [None, "gimp", "sgmp"])
@pytest.mark.parametrize("scheme", ["usf", "musl"])
def test_mass_and_momentum(built, shape, scheme):
    """USF: the step's first momentum transfer; MUSL: the second one."""
    from mpm3d_gb300 import MpmStep
    d = _deck(shape, scheme, False)
    a, b = MpmStep(d, "fp64"), MpmStep(d, "mixed")
    a.run(1)
    b.run(1)
    m = a.download("Mg")
    # (the case is to the point: many sums need more than FP32's bits)
    assert np.sum(m != m.astype(np.float32)) > 50
    np.testing.assert_array_equal(b.download("Mg"), m)
    # (the USF momentum has been integrated, over half a step at the first one:
    # the node velocities, quotients of two FP32 roundings, leave the mixed form
    # some artificial viscosity)
    p = a.download("PXg") + (b.download("FXg") * b.scalars()["CurrentTime"] / 2 if scheme == "usf" else 0.0)
    np.testing.assert_array_max_ulp(b.download("PXg"), p, 1)


@pytest.mark.parametrize("shape", [None, "gimp", "sgmp"])
def test_force(built, shape):
    from mpm3d_gb300 import MpmStep
    d = _deck(shape, "usf", True)
    a, b = MpmStep(d, "fp64"), MpmStep(d, "mixed")
    a.run(1)
    b.run(1)
    f = a.download("FXg")
    assert np.sum(f != f.astype(np.float32)) > 150
    np.testing.assert_array_equal(b.download("FXg"), f)
