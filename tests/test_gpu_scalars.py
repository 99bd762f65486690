"""A caller that observes every step (step(1), then the observables) against
one that steps at once: the same state and observables, bit for bit -- bound
and free particles together, sizes at the edges of the blocks that leave the
partials -- and the asynchronous form of the observables against the waiting
one, two of them in flight."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def mixture(n):
    """About half of the spheres in touching pairs, the rest alone."""
    rng = np.random.default_rng(n)
    per = 12
    k = np.arange(n) // 4 * 2 + (np.arange(n) % 4 == 3)
    p = np.stack([(k % per) * 2.2 - 12.2, (k // per % per) * 2.2 - 12.2, 0.6 + (k // per ** 2) * 2.2], 1)
    p[:, 0] += 0.49 * (np.arange(n) % 4 == 1) - 0.49 * (np.arange(n) % 4 == 0)
    p[:, 0] += 0.05 * (np.arange(n) % 4 == 2)
    p[np.arange(n) % 4 == 2, 2] += 1.05
    return p.reshape(-1), np.full(n, 0.5), 1e-5 * (rng.random(3 * n) - 0.5)


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("n", [1, 255, 256, 257, 1025, 3000])
def test_every_step_observed(dem, wl, n, prec):
    pos, rad, disp = mixture(n)
    pp, pw = wl.material(mu=0.3)
    kw = dict(n=n, world=(30.0, 30.0, 80.0), dt=wl.reduced_dt(5e-7), skin=0.05, precision=prec,
              relist_interval=20)

    def engine():
        e = dem.Engine(**kw)
        e.set_material(pp, pw)
        e.upload(pos, rad, disp, np.zeros(3 * n))
        return e

    a, b = engine(), engine()
    for steps in (7, 13, 23):
        for _ in range(steps):
            a.step(1)
            sa = a.scalars()
        b.step(steps)
        sb = b.scalars()
        assert sa == sb
    if n > 200:
        assert sa["contacts"] > n // 8
    nb = a.scalars_raw_bytes()
    raw = [ctypes.create_string_buffer(nb) for _ in range(2)]
    a.scalars_enqueue(ctypes.addressof(raw[0]))
    a.step(1)
    a.scalars_enqueue(ctypes.addressof(raw[1]))
    a.synchronize()
    assert a.scalars_from_raw(ctypes.addressof(raw[0])) == sa
    assert a.scalars_from_raw(ctypes.addressof(raw[1])) == a.scalars()
    b.step(1)
    for u, v in zip(a.download(), b.download()):
        assert np.array_equal(u, v)
    a.close()
    b.close()
