"""Windows of many small dense components: clusters of five touching spheres
(nine contacts) or ten (twenty-four) among single ones run as cluster batches
as long as a batch's pairs fit a block, however many pairs a bound particle
has; where they do not, as tiles, and a bed always.  The states are those of
the grid-barrier kernel, bit for bit."""
import numpy as np
import pytest

from _cases import dense_lattice

pytestmark = pytest.mark.gpu


def cluster(kind):
    a, s3 = 0.998, np.sqrt(3.0)
    if kind == "ten":
        p = [[(i + j / 2 + k / 2) * a, (j * s3 / 2 + k * s3 / 6) * a, k * np.sqrt(2 / 3) * a]
             for k in range(3) for i in range(3 - k) for j in range(3 - k - i)]
    else:
        t = np.array([[0, 0, 0], [a, 0, 0], [a / 2, a * s3 / 2, 0]])
        h = np.array([0, 0, a * np.sqrt(2 / 3)])
        p = [*t, t.mean(0) + h, t.mean(0) - h]
    return np.array(p) - np.mean(p, 0)


def clusters(dem, wl, kind, sites, every):
    """Every `every`-th site of a wide lattice a cluster, the others a sphere."""
    one = cluster(kind)
    side = int(np.ceil(sites ** (1 / 3)))
    k = np.arange(sites)
    c = np.stack([k % side, k // side % side, k // side ** 2], 1) * 3.6
    c[:, :2] -= c[:, :2].mean(0)
    c[:, 2] += 4
    hit = k % every == 0
    pos = np.concatenate([(c[hit][:, None] + one[None]).reshape(-1, 3), c[~hit]])
    w = dense_lattice(dem, 2, 2, 2)
    w.pos, w.rad, w.n = pos.reshape(-1).copy(), np.full(len(pos), 0.5), len(pos)
    w.world = (side * 3.6 + 2, side * 3.6 + 2, c[:, 2].max() + 8)
    return w


def run(dem, w, prec, steps=60):
    rng = np.random.default_rng(2)
    motion = [1e-5 * (rng.random(3 * w.n) - 0.5) for _ in range(2)]
    e = dem.Engine(**{**w.engine_kwargs(), "precision": prec})
    e.set_material(w.pp, w.pw)
    e.upload(w.pos, w.rad, *motion)
    e.step(steps)
    s, p, work = e.scalars(), e.window_path()["path"], e.window_work()
    out = [*e.download(), *e.pairs(), np.array([s["pairs"], s["contacts"], s["maxhz"]])]
    assert s["status"] == 0
    e.close()
    return out, p, work


# the batches hold 0.3 to 0.9 of what a block can; and more than it can
@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("kind,sites,every,path", [("five", 9000, 8, "batches"), ("five", 40000, 20, "batches"),
                                                   ("ten", 40000, 80, "batches"), ("ten", 3000, 1, "tiles"),
                                                   ("five", 3000, 1, "tiles")])
def test_small_components(dem, wl, cuda, monkeypatch, kind, sites, every, path, prec):
    w = clusters(dem, wl, kind, sites, every)
    a, p, work = run(dem, w, prec)
    assert p == path and work["pairs"] > 1.5 * work["bound"]
    monkeypatch.setenv("DEM_B200_BATCH", "0")
    b, q, _ = run(dem, w, prec)
    assert q == "grid"
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("far", [0, 12000])
def test_a_bed_is_tiles(dem, cuda, prec, far):
    """Also one that is a small part of its system (`far` single spheres above it)."""
    w = dense_lattice(dem, 14, 14, 12)
    if far:
        k = np.arange(far)
        q = np.stack([(k % 9) * 1.3 - 5.2, (k // 9 % 9) * 1.3 - 5.2, 20.0 + (k // 81) * 1.3], 1)
        w.pos = np.concatenate([w.pos, q.reshape(-1)])
        w.rad = np.concatenate([w.rad, np.full(far, 0.5)])
        w.n = w.rad.size
        w.world = (w.world[0], w.world[1], 240.0)
    _, p, work = run(dem, w, prec, steps=100)
    assert p == "tiles" and work["batched"] == 0
