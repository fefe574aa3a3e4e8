"""The fused FP64 field operators against the FP64 oracle, bit for bit, where
their index and quotient rules can go wrong: axes of one, two and three cells
(a node that is its own periodic neighbour), rows longer and shorter than a
block, spacings that are powers of two (exact reciprocals) and not (corrected
quotients), zero and non-zero curls, and odd and even subcycle counts (the
time levels change places)."""
import numpy as np
import pytest

from helpers import oracle_for, periodic_np
from swap_gb300.grid import grd7
from swap_gb300.hybrid import Hybrid, config

pytestmark = pytest.mark.gpu


def _pair(cells, d, ntsub=10, seed=4, flat=False):
    cfg = config(0, cells=cells, ppc=1, seed=seed, ntsub=ntsub, dt=0.002 * ntsub)
    h = Hybrid(cfg, ni_max=cfg.n_particles, coords=grd7(*cfg.nodes, *d))
    h.load_maxwellian()
    rng = np.random.default_rng(seed)
    for n in ("b1", "b12", "b1p2", "bt"):
        a = h.b0 + (0.0 if flat else 0.05) * rng.standard_normal(h.b1.shape)
        getattr(h, n)[...] = periodic_np(a)
    h.np[...] = periodic_np(1.0 + 0.3 * rng.random(h.np.shape))
    for n in ("up", "aj", "E"):
        getattr(h, n)[...] = periodic_np(0.3 * rng.standard_normal(h.up.shape))
    h.nu[...] = 0.01 * rng.random(h.nu.shape)
    h.mark_host_dirty()
    return h, oracle_for(h)


@pytest.mark.parametrize("d", [(1.0, 1.0, 1.0), (0.5, 2.0, 0.25), (0.7, 1.3, 0.9)])
@pytest.mark.parametrize("cells", [(1, 1, 1), (2, 1, 3), (3, 7, 2), (33, 5, 4), (260, 3, 2)])
def test_operators_equal_the_oracle(cells, d):
    h, o = _pair(cells, d, flat=cells == (3, 7, 2))
    dtsub = h.cfg.dt / h.cfg.ntsub
    for x in (h, o):
        x.curlB(x.bt, x.np, x.aj)
        x.edge_to_center(x.bt, x.btc)
        x.get_E(x.E, x.b0, x.bt, x.aj, x.up, x.np, x.nu)
        x.predict_B(x.b0, x.b1, x.b12, x.b1p2, x.bt, x.E, x.aj, x.up, x.np, x.nu, dtsub)
        x.correct_B(x.b0, x.b1, x.b1p2, x.E, x.aj, x.up, x.np, x.nu, dtsub)
    h.sync_to_host()
    for n in ("aj", "bt", "btc", "E", "b1p2"):
        assert np.array_equal(getattr(h, n), getattr(o, n)), n
    h.close()


@pytest.mark.parametrize("d", [(1.0, 1.0, 1.0), (0.7, 1.3, 0.9)])
@pytest.mark.parametrize("cells,ntsub", [((9, 5, 6), 1), ((9, 5, 6), 2), ((1, 3, 2), 3), ((40, 30, 5), 5),
                                         ((64, 64, 40), 2), ((64, 64, 41), 3)])
def test_subcycles_equal_the_entries(cells, ntsub, d):
    """The fused field step (one launch up to 163840 nodes, then one per
    operator) leaves every array as the per-subroutine entries do."""
    h, _ = _pair(cells, d, ntsub)
    r, _ = _pair(cells, d, ntsub)
    h._check(h.lib.swap_field_subcycles(h.ctx))
    dtsub = r.cfg.dt / ntsub
    for _ in range(ntsub):
        r.curlB(r.bt, r.np, r.aj)
        r.predict_B(r.b0, r.b1, r.b12, r.b1p2, r.bt, r.E, r.aj, r.up, r.np, r.nu, dtsub)
        r.correct_B(r.b0, r.b1, r.b1p2, r.E, r.aj, r.up, r.np, r.nu, dtsub)
        r.f_update_tlev(r.b1, r.b12, r.b1p2, r.bt, r.b0)
    for x in (h, r):
        x.sync_to_host()
    for n in ("aj", "bt", "E", "b1", "b12", "b1p2"):
        assert np.array_equal(getattr(h, n), getattr(r, n)), n
    h.close()
    r.close()


def test_courant_violation_takes_the_replayed_count():
    """Above the Courant limit dtsub is halved on the host (gutsf.f:1776-1822);
    the loop launched ahead of that look leaves the state alone."""
    cfg = config(0, cells=(9, 5, 6), ppc=8, seed=4, ntsub=2, dt=2.0)  # dtsub of about twice the Courant time
    x = Hybrid(cfg, ni_max=cfg.n_particles)
    x.load_maxwellian()
    y = oracle_for(x)
    x.ion_step()
    x.sync_to_host()
    y.ion_step()
    for n in ("b1", "b12", "E", "np"):
        a, b = getattr(x, n), getattr(y, n)
        assert np.max(np.abs(a - b)) <= 1e-12 * np.max(np.abs(b)), n
    x.close()
