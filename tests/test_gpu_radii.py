"""The upload's reduction of the radii (largest, solid volume, validity) for
one thread, one block, blocks that stride, twice in a row, from the host and
from the device: the largest and the packing fraction against NumPy (the sum
of at most 2^20 positive terms in blocks: 1e-12 relative)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 255, 257, 1024, 1025, 512 * 1024 + 1])
def test_radii(dem, wl, cuda, n):
    import torch
    rng = np.random.default_rng(n)
    k = np.arange(n)
    pos = np.stack([k % 100 * 2.0 - 99.0, k // 100 % 100 * 2.0 - 99.0, k // 10000 * 2.0 + 1.0], 1).reshape(-1)
    world = (200.0, 200.0, 220.0)
    pp, pw = wl.material()
    e = dem.Engine(n=n, world=world, dt=1e-9, skin=0.05, precision=0)
    e.set_material(pp, pw)
    top = pos.reshape(-1, 3)[:, 2].max()
    for which in ("host", "device", "host"):
        rad = rng.uniform(0.1, 0.5, n)
        if which == "host":
            e.upload(pos, rad)
        else:
            e.upload_device(torch.tensor(pos, device="cuda"), torch.tensor(rad, device="cuda"))
        e.step(1)
        s = e.scalars()
        want = 4 / 3 * np.pi * (rad ** 3).sum() / (world[0] * world[1] * s["maxhz"])
        assert abs(s["maxhz"] - top) < 1e-6 and abs(s["packing_fraction"] - want) <= 1e-12 * want
    for bad in (0.0, -0.3, np.nan):
        rad[n // 2] = bad
        with pytest.raises(dem.DemError, match=f"radius {n // 2} not positive"):
            e.upload(pos, rad)
    e.close()
