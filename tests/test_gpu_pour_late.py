"""A pour set on a context that has stepped already (upload, steps,
dem_set_pour): the particles in the system are fewer than those of the last
re-list, whose outer list and tiles name the others too.  The steps that
follow, as whole windows and one by one, are those of a new context that gets
the same state and the same pour, bit for bit.  Frictionless contacts: a
context's tangential histories, which the new one does not have, are zero."""
import numpy as np
import pytest

from _cases import dense_lattice

pytestmark = pytest.mark.gpu


def _engine(dem, w, prec, mode):
    e = dem.Engine(**{**w.engine_kwargs(), "precision": prec, "force_mode": mode})
    e.set_material({**w.pp, "mu": 0.0}, {**w.pw, "mu": 0.0})
    return e


def _upload(e, torch, w, state, device):
    if device:
        t = [torch.as_tensor(np.ascontiguousarray(v), device="cuda") for v in (state[0], w.rad, state[1], state[2])]
        torch.cuda.synchronize()
        e.upload_device(t[0].data_ptr(), t[1].data_ptr(), t[2].data_ptr(), t[3].data_ptr())
        e.synchronize()
    else:
        e.upload(state[0], w.rad, state[1], state[2])


@pytest.mark.parametrize("chunk", [20, 1])
@pytest.mark.parametrize("device", [True, False])
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("size", [(3, 3, 4), (14, 14, 12)])
def test_pour_after_steps(dem, cuda, prec, mode, device, chunk, size):
    w = dense_lattice(dem, *size)
    n_active = w.n - w.n // 3 - 5
    rng = np.random.default_rng(4)
    start = [w.pos] + [1e-5 * (rng.random(3 * w.n) - 0.5) for _ in range(2)]
    a, b = _engine(dem, w, prec, mode), _engine(dem, w, prec, mode)
    _upload(a, cuda, w, start, device)
    a.step(40)
    _upload(b, cuda, w, a.download(), device)
    out = []
    for e in (a, b):
        e.set_pour(w.n, 1e30, n_active)   # nobody joins
        for _ in range(0, 60, chunk):
            e.step(chunk)
        s = e.scalars()
        assert s["status"] == 0 and e.active_count() == n_active
        out.append([*e.download(), *e.pairs(), np.array([s["pairs"], s["contacts"], s["maxhz"]])])
        e.close()
    assert out[0][3].size and max(out[0][4]) < n_active
    for x, y in zip(*out):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("mode", [0, 1])
def test_layer_after_steps(dem, cuda, mode):
    """As above with a layer that joins in the window's middle: the system
    grows again past the particles it kept."""
    w = dense_lattice(dem, 14, 14, 12)
    n_active = w.n // 2
    layer = w.n - n_active - 7
    a, b = _engine(dem, w, 1, mode), _engine(dem, w, 1, mode)
    zero = np.zeros(3 * w.n)
    _upload(a, cuda, w, [w.pos, zero, zero], True)
    a.step(40)
    _upload(b, cuda, w, a.download(), True)
    out = []
    for e, done in ((a, 40), (b, 0)):
        # due before the 31st step from here (time = dt (step + 1)); the next not before the 61st
        e.set_pour(layer, w.dt * (done + 30.5) * layer / n_active, n_active)
        e.step(60)
        assert e.scalars()["status"] == 0 and e.active_count() == n_active + layer
        out.append([*e.download(), *e.pairs()])
        e.close()
    for x, y in zip(*out):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("mode", [0, 1])
def test_who_joins_again_has_no_history(dem, cuda, prec, mode):
    """With friction: all the particles that a late pour took out join before
    its first step, at the places they had, so their contacts with the others
    are still listed -- and start without history, as in a new context."""
    w = dense_lattice(dem, 14, 14, 12)
    n_active = w.n // 2
    out = []
    a, b = (dem.Engine(**{**w.engine_kwargs(), "precision": prec, "force_mode": mode}) for _ in range(2))
    zero = np.zeros(3 * w.n)
    for e in (a, b):
        e.set_material(w.pp, w.pw)
    _upload(a, cuda, w, [w.pos, zero, zero], True)
    a.step(40)
    _upload(b, cuda, w, a.download(), True)
    for e in (a, b):
        e.set_pour(w.n - n_active, 1e-30, n_active)
        e.step(1)
        assert e.active_count() == w.n and e.scalars()["status"] == 0
        lp, ln, h = e.pairs()
        joined = ln >= n_active
        out.append((lp, ln, np.asarray(h).reshape(-1, 3), joined))
        e.close()
    (lp, ln, h, joined), (lp2, ln2, h2, _) = out
    np.testing.assert_array_equal(lp, lp2)
    np.testing.assert_array_equal(ln, ln2)
    assert joined.any() and (~joined).any() and np.abs(h2[joined]).max() > 0
    np.testing.assert_array_equal(h[joined], h2[joined])
    assert np.abs(h[~joined] - h2[~joined]).max() > 0   # the others kept theirs
