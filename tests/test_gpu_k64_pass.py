"""The FP64 particle passes against the FP64 oracle where their rules can go
wrong: counts that do not fill a warp or a block, ions of one cell in many
warps and of many cells in one, shuffled order, several (mrat, beta_p)
species, spacings that differ from cell to cell, and an open x axis.

The bars are those of test_gpu_parity.py: single-step particle states within
1e-12 of their scale.  Moments and fields here too: a deposit is a sum of at
most a few thousand terms rounded to 1.1e-16 each, divided by a density of
order one.  Grids the oracle has not (its axes are uniform) are compared with
the operator-by-operator form, which the deterministic sums select."""
import numpy as np
import pytest

from conftest import relerr
from helpers import oracle_for, periodic_np
from swap_gb300.grid import grd7
from swap_gb300.hybrid import Hybrid, config

pytestmark = pytest.mark.gpu
TOL = 1e-12


def _stretched(nodes):
    """grd7 with x and z spacings that grow along the axis (initial.f:246-257 for the cells and ratios)."""
    co = grd7(*nodes, 0.9, 1.1, 1.0)
    for q, dg, dc, rat, n in (("qx", "dx_grid", "dx_cell", "xrat", nodes[0]),
                              ("qz", "dz_grid", "dz_cell", "zrat", nodes[2])):
        x = np.cumsum(1.0 + 0.3 * np.arange(n) / n)
        d = np.append(x[1:] - x[:-1], x[-1] - x[-2])
        mid = (x[1:] + x[:-1]) / 2.0
        cell, r = d.copy(), np.full(n, 0.5)
        cell[1:-1] = mid[1:] - mid[:-1]
        r[1:-1] = (x[1:-1] - mid[:-1]) / cell[1:-1]
        for name, v in ((q, x), (dg, d), (dc, cell), (rat, r)):
            getattr(co, name)[...] = v
    return co


def _make(cells, ppc, n=None, shuffle=False, species=False, stretched=False, d=None, sources=False, seed=6,
          dt=0.02):
    cfg = config(1 if sources else 0, cells=cells, ppc=ppc, seed=seed, dt=dt, ntsub=4)
    nmax = cfg.ni_max_hint(8) if sources else cfg.n_particles + 3
    co = _stretched(cfg.nodes) if stretched else (grd7(*cfg.nodes, *d) if d else None)
    h = Hybrid(cfg, ni_max=nmax, coords=co)
    h.load_maxwellian()
    if n is not None:
        h.ni_tot[0] = n
    N = int(h.ni_tot[0])
    rng = np.random.default_rng(seed)
    h.vp1[:N] += 0.02 * rng.standard_normal((N, 3))
    if species:
        heavy = rng.random(N) < 0.3
        h.mrat[:N][heavy] = 1.0 / 16.0
        h.beta_p[:N][heavy] = 3.0
    if shuffle:
        p = rng.permutation(N)
        for a in (h.xp, h.vp, h.vp1, h.mrat, h.beta_p):
            a[:N] = a[:N][p]
    b = h.b0 + 0.05 * rng.standard_normal(h.b1.shape)
    periodic_np(b)
    for name in ("b1", "b12", "b1p2", "bt"):
        getattr(h, name)[...] = b
    if sources:
        h.set_sources(cfg.make_sources())
    h.mark_host_dirty()
    if not stretched:
        return h, oracle_for(h)
    r = Hybrid(cfg, ni_max=nmax, coords=co)
    for name in ("xp", "vp", "vp1", "mrat", "beta_p", "b1", "b12", "b1p2", "bt", "ni_tot"):
        getattr(r, name)[...] = getattr(h, name)
    r.mark_host_dirty()
    r.set_deterministic(True)
    return h, r


@pytest.mark.parametrize("kw", [
    dict(cells=(6, 5, 4), ppc=9),
    dict(cells=(6, 5, 4), ppc=9, shuffle=True, species=True),
    dict(cells=(3, 3, 3), ppc=300, shuffle=True),
    dict(cells=(5, 3, 4), ppc=40, n=60 * 40 - 17),  # a tail that is no whole warp
    dict(cells=(7, 5, 6), ppc=8, d=(0.7, 1.3, 0.9)),
    dict(cells=(7, 5, 6), ppc=8, stretched=True),
    dict(cells=(7, 5, 6), ppc=8, stretched=True, shuffle=True, species=True),
])
def test_step_equals_the_oracle(kw):
    h, o = _make(**kw)
    h.run(2)
    h.sync_to_host()
    for _ in range(2):
        o.ion_step()
    if isinstance(o, Hybrid):
        o.sync_to_host()
    N = int(h.ni_tot[0])
    for name in ("xp", "vp", "vp1"):
        assert relerr(getattr(h, name)[:N], getattr(o, name)[:N]) < TOL, name
    for name in ("np", "up", "b1", "E", "btc", "aj"):
        assert relerr(getattr(h, name), getattr(o, name)) < TOL, name
    # the COMMON weights a later entry reads are those of maind.f:411
    want = h.np.copy()
    h.update_np(h.np)
    h.sync_to_host(h.np)
    assert relerr(h.np, want) < 1e-13
    h.close()


def test_halves_of_the_step_and_open_x():
    """swap_ion_step_pre/_post take the move of maind.f:479 apart; with an open
    x axis one removal after both half moves takes the ions that two did."""
    h, o = _make((12, 4, 4), 12, sources=True, dt=0.05)
    r, _ = _make((12, 4, 4), 12, sources=True, dt=0.05)
    h.run(3)
    for _ in range(3):
        for entry in ("swap_ion_step_pre", "swap_field_subcycles", "swap_ion_step_post"):
            r._check(getattr(r.lib, entry)(r.ctx))
    for x in (h, r):
        x.sync_to_host()
    N = int(h.ni_tot[0])
    assert N == int(r.ni_tot[0]) and N != h.cfg.n_particles
    for name in ("xp", "vp", "vp1", "mrat", "beta_p"):
        assert relerr(getattr(h, name)[:N], getattr(r, name)[:N]) < TOL, name
    h.close()
    r.close()


def test_an_ion_outside_the_grid_is_reported():
    h, _ = _make((6, 5, 4), 4)
    from swap_gb300 import abi
    for bad in (np.nan, -3.0, 1e300):
        keep = h.xp.copy(order="F")
        h.xp[5, 0] = bad
        h.mark_host_dirty(h.xp)
        with pytest.raises(abi.SwapError, match="EDOMAIN"):
            h.ion_step()
        h.xp[...] = keep
        h.mark_host_dirty()
        h.ion_step()
    h.close()
