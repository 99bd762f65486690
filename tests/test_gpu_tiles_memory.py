"""The tiles' memory: a context takes it when a window first needs tiles, goes
without when the device is full, and gives it back to a later call that needs
the room -- with the same states bit for bit."""
import numpy as np
import pytest

from _cases import dense_lattice

pytestmark = pytest.mark.gpu
MIB = 1 << 20


def engine(dem, w, prec, mode=0):
    e = dem.Engine(**{**w.engine_kwargs(), "precision": prec, "force_mode": mode})
    e.set_material(w.pp, w.pw)
    return e


def free(torch):
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def fill(torch, leave):
    """Takes the device's free memory but `leave` bytes."""
    out = []
    for step in (1 << 30, 64 * MIB, 2 * MIB):
        n = (free(torch) - leave) // step
        if n > 0:
            out.append(torch.empty(n * step, dtype=torch.uint8, device="cuda"))
    return out


def gas(dem, wl, n=400_000):
    w = wl.rsa_500k(n=n, box=(100.0, 100.0, 320.0))
    assert w.n == n
    return w


@pytest.mark.parametrize("prec", [0, 1])
def test_a_gas_holds_none(dem, wl, cuda, monkeypatch, prec):
    w = gas(dem, wl)
    used = {}
    for batch in ("1", "0", "1", "0"):   # the first two load the kernels
        monkeypatch.setenv("DEM_B200_BATCH", batch)
        before = free(cuda)
        e = engine(dem, w, prec)
        e.upload(w.pos, w.rad)
        e.step(60)
        assert e.scalars()["status"] == 0
        assert e.window_path()["path"] == ("batches" if batch == "1" else "grid")
        used[batch] = before - free(cuda)
        e.close()
    # the components' arrays (10 words a particle), allocation granularity
    assert used["1"] - used["0"] <= 40 * w.n + 16 * MIB, used


@pytest.mark.parametrize("prec", [0, 1])
def test_tiles_come_with_the_first_dense_windows(dem, wl, cuda, prec):
    """A context that was used for a gas, then gets a bed: in one call."""
    bed = dense_lattice(dem, 44, 44, 40)
    thin = dense_lattice(dem, 44, 44, 40, spacing=1.2)   # nothing in contact
    world = tuple(max(a, b) for a, b in zip(bed.world, thin.world))
    bed.world = thin.world = world
    new, used = engine(dem, bed, prec), engine(dem, thin, prec)
    used.upload(thin.pos, thin.rad)
    used.step(60)
    assert used.window_path()["path"] == "batches"
    for e in (new, used):
        e.upload(bed.pos, bed.rad)
        e.step(60 * 20)
        assert e.scalars()["status"] == 0 and e.window_path()["path"] == "tiles"
    for x, y in zip(new.download(), used.download()):
        np.testing.assert_array_equal(x, y)
    new.close()
    used.close()


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("prec", [0, 1])
def test_a_full_device(dem, cuda, prec, mode):
    """No room for the tiles; and a context with tiles, whose next allocation
    finds no room until they are given back."""
    w = dense_lattice(dem, 60, 60, 50)
    first = engine(dem, w, prec, mode)   # with tiles; loads the kernels
    first.upload(w.pos, w.rad)
    first.step(60)
    first.record_forces(True)
    first.step(1)
    first.record_forces(False)
    first.close()
    first, late = engine(dem, w, prec, mode), engine(dem, w, prec, mode)
    first.upload(w.pos, w.rad)
    first.step(20)
    assert first.window_path()["path"] == "tiles"
    late.upload(w.pos, w.rad)
    held = fill(cuda, 6 * MIB)
    late.step(20)
    if mode == 0:
        assert late.window_path()["path"] == "grid"
    first.record_forces(True)    # 13 words a particle: more than is left
    first.record_forces(False)
    first.step(40)
    assert first.window_path()["path"] == "grid"
    late.step(40)
    del held
    cuda.cuda.empty_cache()
    for e in (first, late):
        assert e.scalars()["status"] == 0
    a, b = first.download() + first.pairs(), late.download() + late.pairs()
    first.close()
    late.close()
    ref = engine(dem, w, prec, mode)
    ref.upload(w.pos, w.rad)
    ref.step(60)
    for x, y, z in zip(a, b, ref.download() + ref.pairs()):
        np.testing.assert_array_equal(x, z)
        np.testing.assert_array_equal(y, z)
    ref.close()
