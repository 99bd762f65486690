"""Windows whose components do not fit a block, stepped as tiles
(csrc/dem_tile.cuh), against the grid-barrier window kernel
(DEM_B200_BATCH=0), in PP mode against the per-step kernels
(DEM_B200_WINDOW=0): the same states, pair lists with their histories and
observables, bit for bit -- one tile, tiles that stay in shared memory, blocks
that stream several tiles or have one while others have two, long rows (a
close-packed crystal), a density so uneven that the first window's tiles do
not fit and later ones are smaller, short windows, and the adjoint's tape."""
import numpy as np
import pytest

from _cases import dense_lattice

pytestmark = pytest.mark.gpu


def crystal(dem, wl, nx, ny, nz, loose=0):
    """Face-centred cubic spheres (12 neighbours each) under slight overlap in
    a wide box, and `loose` touching pairs of spheres high above."""
    rng = np.random.default_rng(3)
    a = np.sqrt(2.0) * 0.9985
    base = np.array([[0, 0, 0], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]])
    cell = np.stack(np.meshgrid(np.arange(nx), np.arange(ny), np.arange(nz), indexing="ij"), -1).reshape(-1, 1, 3)
    p = ((cell + base[None]) * a).reshape(-1, 3)
    p[:, :2] -= p[:, :2].mean(0)
    p[:, 2] += 0.52
    side = max(24.0, np.abs(p[:, :2]).max() * 2 + 4)
    if loose:
        per = int(side / 2.5) - 1
        k = np.arange(loose)
        q = np.stack([(k % per) * 2.5 - side / 2 + 1.5, (k // per % per) * 2.5 - side / 2 + 1.5,
                      p[:, 2].max() + 3 + (k // per ** 2) * 1.5], 1)
        p = np.concatenate([p, q, q + [0.998, 0, 0]])
    n = p.shape[0]
    rad = rng.uniform(0.4995, 0.5005, n).astype(np.float32).astype(np.float64)
    pp, pw = wl.material(mu=0.3, roll_rel=0.002)
    return wl.Workload("crystal", n, p.reshape(-1).copy(), rad, (side, side, p[:, 2].max() + 10), wl.reduced_dt(5e-7),
                       60, 20, 0.05, dem.PREC_FP64, pp, pw)


def run(dem, w, prec, K, steps, motion, adjoint=0, mode=0):
    e = dem.Engine(**{**w.engine_kwargs(), "precision": prec, "relist_interval": K, "force_mode": mode})
    e.set_material(w.pp, w.pw)
    e.upload(w.pos, w.rad, *motion)
    if adjoint:
        g = e.adjoint(steps, adjoint, dem.OBJ_POTENTIAL)
        out = [g["d_radii"], np.array(list(g["d_pp"].values()) + list(g["d_pw"].values()) + [g["value"]])]
    else:
        e.step(steps)
        out = list(e.pairs())
    s = e.scalars()
    work = e.window_work()
    out += list(e.download())
    e.close()
    return out, [s[k] for k in ("pairs", "contacts", "maxhz", "status")], work


def check(dem, w, prec, monkeypatch, K=20, steps=60, adjoint=0, mode=0):
    rng = np.random.default_rng(9)
    motion = [1e-5 * (rng.random(3 * w.n) - 0.5) for _ in range(2)]
    a, sa, work = run(dem, w, prec, K, steps, motion, adjoint, mode)
    switch = "DEM_B200_WINDOW" if mode else "DEM_B200_BATCH"
    monkeypatch.setenv(switch, "0")
    b, sb, _ = run(dem, w, prec, K, steps, motion, adjoint, mode)
    monkeypatch.delenv(switch)
    assert work["batched"] == (-1 if mode else 0) and sa[3] == 0
    assert sa == sb
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("size", [(12, 12, 3), (14, 14, 12), (37, 31, 9), (44, 44, 40)])
def test_lattice(dem, cuda, monkeypatch, prec, size):
    """From a dozen tiles to blocks that stream two and more (77,440 spheres:
    more than the resident blocks hold in either precision)."""
    check(dem, dense_lattice(dem, *size), prec, monkeypatch)


@pytest.mark.parametrize("K", [2, 3])
def test_short_windows(dem, cuda, monkeypatch, K):
    check(dem, dense_lattice(dem, 14, 14, 12), 1, monkeypatch, K=K, steps=12 * K)


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("size,loose", [((10, 10, 5), 0), ((26, 26, 12), 0), ((24, 24, 20), 20000)])
def test_crystal(dem, wl, cuda, monkeypatch, prec, size, loose):
    check(dem, crystal(dem, wl, *size, loose=loose), prec, monkeypatch, steps=100)


@pytest.mark.parametrize("prec", [0, 1])
def test_adjoint_tape(dem, cuda, monkeypatch, prec):
    check(dem, dense_lattice(dem, 14, 14, 12), prec, monkeypatch, steps=40, adjoint=20)


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("K", [2, 3, 20])
def test_pp(dem, cuda, monkeypatch, prec, K):
    """The particle-parallel mode, an odd and an even number of steps per
    window (the state and history buffers alternate)."""
    check(dem, dense_lattice(dem, 14, 14, 12), prec, monkeypatch, K=K, steps=5 * K, mode=1)


@pytest.mark.parametrize("prec", [0, 1])
def test_pp_large_and_uneven(dem, wl, cuda, monkeypatch, prec):
    check(dem, dense_lattice(dem, 44, 44, 40), prec, monkeypatch, steps=40, mode=1)
    check(dem, crystal(dem, wl, 24, 24, 20, loose=20000), prec, monkeypatch, steps=60, mode=1)


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("mode", [0, 1])
def test_mostly_free(dem, wl, cuda, monkeypatch, prec, mode):
    """A small crystal under a dilute cloud: few bound particles among many,
    and none at all."""
    w = crystal(dem, wl, 14, 14, 12)
    rng = np.random.default_rng(5)
    k = np.arange(30000)
    cloud = np.stack([(k % 30) * 2.0 - 29, (k // 30 % 30) * 2.0 - 29, 30 + (k // 900) * 2.0], 1)
    cloud += rng.uniform(-0.3, 0.3, cloud.shape)
    w.pos = np.concatenate([w.pos, cloud.reshape(-1)])
    w.rad = np.concatenate([w.rad, np.full(k.size, 0.5)])
    w.n = w.rad.size
    w.world = (64.0, 64.0, 120.0)
    check(dem, w, prec, monkeypatch, steps=60, mode=mode)
    if mode:
        w.pos, w.rad, w.n = w.pos[-3 * k.size:].copy(), w.rad[-k.size:].copy(), k.size
        check(dem, w, prec, monkeypatch, steps=40, mode=mode)
