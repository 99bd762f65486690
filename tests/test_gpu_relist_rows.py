"""The re-list's rows against all pairs by NumPy: rows and reverse rows of every
length about the two register sorts and the kept candidates (7-9, 15-17, 40),
mixed within a warp, and particle counts at the edges of the candidate pass's
tiles, one particle per thread and four."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def groups(n, rng):
    """Groups of 1 to 41 tiny spheres within 0.68 of one another, 1.9 apart
    from the next group, in a shuffled order of ids."""
    size, pts, gid, g = [1, 2, 8, 9, 10, 11, 16, 17, 18, 19, 41, 3, 1, 1, 5], [], [], 0
    while len(gid) < n:
        m = min(size[g % len(size)] if n < 4000 else 1 + 2 * (g % 17 == 0), n - len(gid))
        c = np.array([g % 60, g // 60 % 60, g // 3600]) * 1.9 + [-57.0, -57.0, 1.0]
        d = rng.normal(size=(m, 3))
        d *= 0.34 * rng.random((m, 1)) ** (1 / 3) / np.linalg.norm(d, axis=1, keepdims=True)
        pts.append(c + d)
        gid += [g] * m
        g += 1
    p, gid = np.concatenate(pts), np.array(gid)
    o = rng.permutation(n)
    return p[o], gid[o]


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("n", [511, 512, 513, 2048, 2049, (1 << 18) - 1, 1 << 18, (1 << 18) + 1])
def test_rows(dem, wl, n, prec):
    rng = np.random.default_rng(n)
    p, gid = groups(n, rng)
    pp, pw = wl.material(mu=0.3)
    e = dem.Engine(n=n, world=(120.0, 120.0, 200.0), dt=1e-6, skin=0.7, precision=prec, relist_interval=20, cell=0.8,
                   pair_capacity=40 * n if n < 4000 else 8 * n)
    e.set_material(pp, pw)
    e.upload(p.reshape(-1), np.full(n, 0.01))
    for _ in range(2):   # the second list carries from the first
        e.step(20)
        lp, ln = e.pairs()[:2]
        o = np.argsort(gid, kind="stable")   # groups together, ids ascending
        same = [(o[:-d], o[d:], gid[o[:-d]] == gid[o[d:]]) for d in range(1, 41)]
        want = np.concatenate([np.stack([a[m], b[m]], 1) for a, b, m in same])
        want = want[np.lexsort((want[:, 1], want[:, 0]))]
        assert np.array_equal(np.stack([lp, ln], 1).astype(np.int64), want)
    assert e.scalars()["status"] == 0
    e.close()
