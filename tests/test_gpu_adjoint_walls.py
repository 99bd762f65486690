"""The reverse step where many particles touch a wall and few pairs are listed
(csrc/dem_adjoint.cu gives the walls a thread per particle then): against the
particle-parallel form, and without rounds of particles after one another.
Both reverse the same FP64 tape and differ in the order of sums, as in the
tests of the two forms: 1e-9 of each output's norm."""
import numpy as np
import pytest

from _cases import dense_lattice

pytestmark = pytest.mark.gpu


def floor_layer(dem, n, pairs):
    """n spheres on the floor, apart from one another but for `pairs` touching pairs."""
    w = dense_lattice(dem, 2, 2, 2)
    side = int(np.ceil(np.sqrt(n)))
    k = np.arange(n)
    p = np.stack([(k % side) * 1.6, (k // side) * 1.6, np.full(n, 0.4995)], 1)
    p[:, :2] -= p[:, :2].mean(0)
    odd = k[(k % side) % 2 == 1][:pairs]   # moved to the sphere on its left
    p[odd, 0] -= 0.602
    w.pos, w.rad, w.n = p.reshape(-1).copy(), np.full(n, 0.5), n
    w.world = (side * 1.6 + 4, side * 1.6 + 4, 20.0)
    return w


def reverse(dem, w, prec, reps=1):
    rng = np.random.default_rng(8)
    motion = [rng.normal(0, 3e-6, 3 * w.n), rng.normal(0, 3e-5, 3 * w.n)]
    e = dem.Engine(**{**w.engine_kwargs(), "precision": prec})
    e.set_material(w.pp, w.pw)
    ms = []
    for _ in range(reps):
        e.upload(w.pos, w.rad, *motion)
        g = e.adjoint(200, 100, dem.OBJ_POTENTIAL)
        ms.append(g["adjoint_ms"])
    assert e.scalars()["status"] == 0 and e.window_work()["wall_candidates"] == w.n
    e.close()
    return [np.asarray(g["d_radii"]), np.array(list(g["d_pp"].values())), np.array(list(g["d_pw"].values()))], min(ms)


# one block of walls; about the sixteenth of the grid that a bed's walls get;
# more; more than the grid has threads
@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("n,pairs", [(100, 20), (2400, 0), (2600, 500), (9000, 1500), (60000, 20000)])
def test_forms_agree(dem, cuda, monkeypatch, n, pairs, prec):
    w = floor_layer(dem, n, pairs)
    a, _ = reverse(dem, w, prec)
    monkeypatch.setenv("DEM_B200_ADJ", "pp")
    b, _ = reverse(dem, w, prec)
    for u, v in zip(a, b):
        assert np.isfinite(v).all()
        assert np.linalg.norm(u - v) <= 1e-9 * max(np.linalg.norm(v), 1e-12)


def test_walls_are_one_round(dem, cuda):
    """Nine thousand particles on the floor reverse in little more than the
    time of one thousand: both are one round of threads."""
    # 1.68 times with a sixteenth of the blocks for the walls
    few, many = (reverse(dem, floor_layer(dem, n, 300), 1, reps=5)[1] for n in (1000, 9000))
    assert many < 1.5 * few, (few, many)
