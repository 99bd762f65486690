"""The compatible neighbour rows and pair forces at the edges of their
warps: rows of up to 120 entries (past a warp's list of 96), rows cut at the
caller's length, particle and pair counts about 32, and arrays aligned to
eight bytes only."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CUB = 1.2


def rows(dem, torch, pos, n, maxppc, error=False):
    c = dem.compat
    lo = pos.min(0) - 0.1
    grid = tuple(int(v) for v in np.ceil((pos.max(0) - lo + 0.1) / CUB).astype(int))
    w = lambda k: torch.zeros(k, dtype=torch.int32, device="cuda")   # noqa: E731
    p = torch.tensor(pos.reshape(-1), device="cuda")
    h0, h1, start, anei, ng, nl = w(2 * n), w(2 * n), w(int(np.prod(grid))), w(n * maxppc), w(n), w(n)
    c.set_cutoff(1.0, CUB)
    c.calcHash(p, h0, grid, (CUB,) * 3, tuple(lo), n)
    c.RadixSort(h0, h1, n, 32)
    c.findCellStart(h0, start, n, start.numel())
    args = (p, h0, start, grid, (CUB,) * 3, tuple(lo), maxppc, n, anei, ng, nl)
    if error:
        with pytest.raises(dem.DemError):
            c.neighborarray(*args)
    else:
        c.neighborarray(*args)
    torch.cuda.synchronize()
    return anei.cpu().numpy().reshape(n, maxppc), ng.cpu().numpy(), nl.cpu().numpy()


@pytest.mark.parametrize("n,side", [(1, 1.0), (31, 2.0), (32, 2.0), (33, 2.0), (120, 1.2), (700, 3.5), (1000, 6.0)])
def test_rows(dem, cuda, n, side):
    import torch
    pos = np.random.default_rng(n).random((n, 3)) * side
    d = pos[None] - pos[:, None]
    near = (d[..., 0] * d[..., 0] + d[..., 1] * d[..., 1] + d[..., 2] * d[..., 2] < CUB * CUB) & ~np.eye(n, dtype=bool)
    want = [np.flatnonzero(r) for r in near]
    longest = max(len(r) for r in want)
    if n == 120:
        assert longest > 96
    anei, ng, nl = rows(dem, torch, pos, n, longest + 3)
    for i, r in enumerate(want):
        up, dn = r[r > i], r[r < i]
        assert (ng[i], nl[i]) == (up.size, dn.size)
        assert np.array_equal(anei[i], np.concatenate([up, dn, np.full(longest + 3 - r.size, -1)]))
    if longest > 4:   # rows cut: as many as fit, all of them neighbours, the rest empty
        cut = longest - 2
        anei, ng, nl = rows(dem, torch, pos, n, cut, error=True)
        for i, r in enumerate(want):
            k = min(cut, r.size)
            assert ng[i] + nl[i] == k and ng[i] == min(cut, (r > i).sum())
            assert np.isin(anei[i, :k], r).all() and np.unique(anei[i, :k]).size == k and (anei[i, k:] == -1).all()


@pytest.mark.parametrize("total", [1, 31, 32, 33, 255, 257])
def test_pair_forces_of_any_alignment(dem, cuda, total):
    """The same pairs from arrays at an odd multiple of eight bytes and from
    aligned ones: the same bits; nothing is written past the last pair."""
    import torch
    rng = np.random.default_rng(total)
    n = 2 * total
    pos = np.zeros((n, 3))
    pos[0::2, 0] = pos[1::2, 0] = 3.0 * np.arange(total)
    pos[1::2] += rng.normal(size=(total, 3)) * [0.3, 0.3, 0.3] + [0.75, 0.0, 0.0]
    dem.compat.set_material(dict(estarp=1e6, ufricp=0.3, vpois=0.3, dampnp=0.3, damptp=0.3, upp=5e-4),
                            dict(estarw=1e6, ufricw=0.3, vpoisw=0.3, dampnw=0.3, damptw=0.3, upw=5e-4))
    disp, rot, hist = (1e-5 * rng.normal(size=(k, 3)) for k in (n, n, total))
    out = []
    for shift in (0, 1):
        def at(v, shift=shift):
            t = torch.full((v.size + 8,), 7.0, dtype=torch.float64, device="cuda")
            t[shift:shift + v.size] = torch.tensor(np.ascontiguousarray(v).reshape(-1), device="cuda")
            return t, t[shift:]
        w = lambda v: torch.tensor(np.asarray(v, dtype=np.int32), device="cuda")   # noqa: E731
        x, d, a, r, m = (at(v)[1] for v in (pos, disp, rot, np.full(n, 0.5), np.full(n, 1.0)))
        lp, ln, oln, cp = w(2 * np.arange(total)), w(2 * np.arange(total) + 1), w(np.zeros(total)), w(np.zeros(total))
        full = [at(v) for v in (hist, np.zeros(total), 0 * hist, np.zeros(total), 0 * hist, 0 * hist, 0 * hist)]
        h, fr, oh, ofr, f, ti, tj = (t[1] for t in full)
        dem.compat.calculateforcepair(x, d, a, r, m, lp, ln, oln, h, fr, oh, ofr, 1e-3, f, ti, tj, cp, total)
        torch.cuda.synchronize()
        for whole, view in full:
            size = view.numel() - 8 + shift
            assert (whole[:shift] == 7).all() and (whole[shift + size:] == 7).all()
        out.append([t[:k].cpu().numpy() for t, k in ((h, 3 * total), (fr, total), (oh, 3 * total), (ofr, total),
                                                     (f, 3 * total), (ti, 3 * total), (tj, 3 * total), (cp, total))])
    for u, v in zip(*out):
        assert np.array_equal(u, v)
    touching = np.linalg.norm(pos[1::2] - pos[0::2], axis=1) < 1.0
    assert np.array_equal(out[0][-1] != 0, touching)
    assert (out[0][4].reshape(-1, 3)[~touching] == 0).all() and np.abs(out[0][4].reshape(-1, 3)[touching]).sum(1).all()
