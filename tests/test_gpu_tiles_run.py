"""Which windows run as tiles (csrc/dem_tile.cuh), as dem_window_path reports
it: dense windows do, in the batched and the particle-parallel mode and while
the adjoint writes its tape, with more tiles than blocks where the system is
large.  And tiles around a sphere with a long row, bit for bit those of the
kernels they replace."""
import numpy as np
import pytest

from _cases import dense_lattice
from test_gpu_tiles import check, crystal

pytestmark = pytest.mark.gpu


def engine(dem, w, prec, mode=0, K=20, **kw):
    e = dem.Engine(**{**w.engine_kwargs(), "precision": prec, "force_mode": mode, "relist_interval": K, **kw})
    e.set_material(w.pp, w.pw)
    e.upload(w.pos, w.rad)
    return e


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("size", [(12, 12, 3), (14, 14, 12), (37, 31, 9), (44, 44, 40)])
def test_dense_windows_are_tiles(dem, cuda, prec, mode, size):
    w = dense_lattice(dem, *size)
    e = engine(dem, w, prec, mode)
    assert e.window_path()["path"] == "steps"
    e.step(40)
    p = e.window_path()
    bound = e.window_work()["bound"]
    e.close()
    assert p["path"] == "tiles" and p["shrink"] == 0 and p["blocks"] <= p["tiles"]
    assert (p["tiles"] - 1) * p["tile_size"] < bound <= p["tiles"] * p["tile_size"]
    assert (p["tiles"] > p["blocks"]) == (size[0] == 44)   # blocks that stream several tiles


@pytest.mark.parametrize("K", [2, 3])
def test_short_windows_are_tiles(dem, cuda, K):
    e = engine(dem, dense_lattice(dem, 14, 14, 12), 1, K=K)
    e.step(4 * K)
    assert e.window_path()["path"] == "tiles"
    e.close()


def test_the_adjoint_runs_on_tiles(dem, cuda):
    e = engine(dem, dense_lattice(dem, 14, 14, 12), 1)
    e.adjoint(40, 20, dem.OBJ_POTENTIAL)
    assert e.window_path()["path"] == "tiles"
    e.close()


def test_few_pairs_are_batches(dem, wl, cuda):
    e = engine(dem, crystal(dem, wl, 1, 1, 1, loose=3000), 0)
    e.step(40)
    assert e.window_work()["batched"] == 1 and e.window_path()["path"] == "batches"
    e.close()


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("mode", [0, 1])
def test_long_row(dem, cuda, monkeypatch, prec, mode):
    """A sphere of eight times the others' size in a bed of them, and a thick
    skin: a row of some 170 entries, in several tiles."""
    w = dense_lattice(dem, 20, 20, 16)
    p = w.pos.reshape(-1, 3)
    c = np.array([0.0, 0.0, 8.0])
    keep = np.linalg.norm(p - c, axis=1) > 4.0 + w.rad - 0.001
    w.pos = np.concatenate([p[keep], [c]]).reshape(-1).copy()
    w.rad = np.concatenate([w.rad[keep], [4.0]])
    w.n = w.rad.size
    w.skin = 0.6
    w.pair_capacity = 16 * w.n
    e = engine(dem, w, prec, mode)
    e.step(40)
    assert e.window_path()["path"] == "tiles" and e.scalars()["max_row"] > 96
    e.close()
    check(dem, w, prec, monkeypatch, steps=60, mode=mode)


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("mode", [0, 1])
def test_an_upload_starts_over(dem, wl, cuda, prec, mode):
    """A state whose tiles do not fit, then an even one in the same context:
    its tiles are those of a new context from the first window on."""
    even = dense_lattice(dem, 44, 44, 40)
    uneven = crystal(dem, wl, 14, 14, 12, loose=(even.n - 14 * 14 * 12 * 4) // 2)
    assert uneven.n == even.n
    even.world = tuple(max(a, b) for a, b in zip(even.world, uneven.world))
    uneven.world = even.world
    new = engine(dem, even, prec, mode)
    new.step(20)
    used = engine(dem, uneven, prec, mode)
    used.step(100)
    assert used.window_path()["path"] == "grid" and used.window_path()["shrink"] > 1
    used.upload(even.pos, even.rad)
    used.step(20)
    p = used.window_path()
    assert p == new.window_path() and p["path"] == "tiles" and p["shrink"] == 0
    for x, y in zip(new.download(), used.download()):
        np.testing.assert_array_equal(x, y)
    new.close()
    used.close()


def test_larger_tiles_are_tried_again(dem, wl, cuda):
    """In one run: the shrink that a window left is lowered after a number of
    windows, not kept for good."""
    e = engine(dem, crystal(dem, wl, 14, 14, 12, loose=30000), 0, K=2)
    seen = []
    for _ in range(260):
        e.step(2)
        seen.append(e.window_path()["shrink"])
    e.close()
    assert max(seen) > 0 and any(b < a for a, b in zip(seen, seen[1:])), seen
