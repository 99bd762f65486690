"""The two-phase reverse step against the particle-parallel one
(DEM_B200_ADJ=pp, the library's quotients and roots throughout): from one
sphere to blocks that sort several rounds of pairs, with constants and states
at which the branch-free quotients and roots are left for the library's
(frictionless, very soft, no rolling, no rotation).  Both reverse the same
FP64 tape; they differ in the order of FP64 sums of at most ~10^4 terms, whose
cancellation in these cases is below 10^3: 1e-9 of each output's norm."""
import numpy as np
import pytest

from _cases import dense_lattice

pytestmark = pytest.mark.gpu

KINDS = {"ordinary": {}, "frictionless": dict(mu=0.0), "soft": dict(estar=1e-4), "no rolling": dict(roll_rel=0.0),
         "still": {}}


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("kind", list(KINDS))
@pytest.mark.parametrize("size", [(1, 1, 1), (2, 1, 1), (5, 5, 3), (20, 20, 12)])
def test_forms_agree(dem, monkeypatch, size, kind, prec):
    w = dense_lattice(dem, nx=size[0], ny=size[1], nz=size[2], seed=3)
    w.pos.reshape(-1, 3)[:, 2] -= 5e-4
    rng = np.random.default_rng(12)
    move = 0.0 if kind == "still" else 1.0
    pdis, angv = move * rng.normal(0, 3e-6, 3 * w.n), move * rng.normal(0, 3e-5, 3 * w.n)
    pp, pw = ({**c, **KINDS[kind]} for c in (w.pp, w.pw))
    out = []
    for flag in ("pair", "pp"):
        monkeypatch.setenv("DEM_B200_ADJ", flag) if flag == "pp" else monkeypatch.delenv("DEM_B200_ADJ", False)
        e = dem.Engine(**{**w.engine_kwargs(), "precision": prec})
        e.set_material(pp, pw)
        e.upload(w.pos, w.rad, pdis, angv)
        g = e.adjoint(40, 20, dem.OBJ_POTENTIAL)
        out.append([np.asarray(g["d_radii"]), np.array(list(g["d_pp"].values())), np.array(list(g["d_pw"].values()))])
        assert e.scalars()["status"] == 0
        e.close()
    for u, v in zip(*out):
        assert np.isfinite(v).all()
        assert np.linalg.norm(u - v) <= 1e-9 * max(np.linalg.norm(v), 1e-12)
