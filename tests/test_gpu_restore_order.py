"""Host data that enters a context goes through its stream: behind the steps
that still run and before the kernels that read it. A restart image of the mixed
form that carries no momentum bound (as USF scenes' images once did) has its
bound taken from the restored particles by a kernel that follows at once."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ["Xp", "VXp", "SM", "SD", "PXg"]


@pytest.mark.parametrize("shape,n", [(None, 5), ("gimp", 9), ("bimp", 16), ("sgmp", 30)])
def test_image_without_momentum_bound(built, tmp_path, shape, n):
    from mpm3d_gb300 import Deck, MpmStep, decks
    d = Deck.parse(decks.generic_block("1 elas 1000 1e6 0.3", counts=(n, n, n), shape=shape, velocity=(1.0, 0.5, -5.0)))
    a = MpmStep(d, "mixed")
    a.run(6)
    path = tmp_path / "image"
    a.save(str(path))
    a.run(4)
    want = [a.download(f) for f in FIELDS]
    # the four bounds of the scene's state (single precision, mass first)
    img = bytearray(path.read_bytes())
    mass = np.float32(d.particles()["mass"].max()).tobytes()
    at = img.find(mass, 0, 4096)
    assert at > 0 and img.find(mass, at + 4, at + 64) < 0
    bounds = np.frombuffer(bytes(img[at:at + 16]), dtype=np.float32)
    assert np.all(bounds > 0), bounds
    img[at + 12:at + 16] = bytes(4)
    path.write_bytes(img)
    for _ in range(10):
        b = MpmStep(d, "mixed")
        b.load(str(path))
        b.run(4)
        for f, w in zip(FIELDS, want):
            np.testing.assert_array_equal(b.download(f), w, err_msg=f"{shape} {f}")


@pytest.mark.parametrize("form", ["fp64", "mixed"])
@pytest.mark.parametrize("shape", [None, "gimp", "sgmp"])
def test_load_behind_running_steps(built, tmp_path, form, shape):
    """A load called while steps are still running discards them."""
    from mpm3d_gb300 import Deck, MpmStep, decks
    d = Deck.parse(decks.generic_block("1 elas 1000 1e6 0.3", counts=(16, 16, 16), shape=shape, velocity=(1.0, 0.5, -5.0)))
    a = MpmStep(d, form)
    a.run(6)
    a.save(str(tmp_path / "image"))
    a.run(5)
    want = [a.download(f) for f in FIELDS]
    for _ in range(3):
        a.run(300)
        a.load(str(tmp_path / "image"))
        a.run(5)
        for f, w in zip(FIELDS, want):
            np.testing.assert_array_equal(a.download(f), w, err_msg=f"{form} {shape} {f}")


@pytest.mark.parametrize("shape", [None, "gimp"])
def test_upload_behind_running_steps(built, shape):
    from mpm3d_gb300 import Deck, MpmStep, decks
    d = Deck.parse(decks.generic_block("1 elas 1000 1e6 0.3", counts=(16, 16, 16), shape=shape, velocity=(1.0, 0.5, -5.0)))
    a, b = MpmStep(d, "fp64"), MpmStep(d, "fp64")
    v = d.particles()["VXp"] * 1.5
    for m, wait in ((a, True), (b, False)):
        m.run(100)
        if wait:
            m.sync()
        m.upload("VXp", v)
        m.run(5)
    for f in FIELDS:
        np.testing.assert_array_equal(a.download(f), b.download(f), err_msg=f"{shape} {f}")
