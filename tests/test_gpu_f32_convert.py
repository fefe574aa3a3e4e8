"""The FP32 form's conversions, in (f32_begin) and out (f32_end), against numpy:
the cell rules and offsets of positions on and beside the nodes, on unit and
other spacings, and the rounding of velocities at ties, zeros, denormals and
the largest floats.  Cells and velocities are exact; a position comes back
within the rounding of q(1) + (cell + offset) * d in 64 bits."""
import numpy as np
import pytest

from swap_gb300.grid import grd7
from swap_gb300.hybrid import Hybrid, config

pytestmark = pytest.mark.gpu

T24 = 2.0**-24
SPEEDS = np.array([0.0, -0.0, 1.0 + T24, 1.0 + 3 * T24, -(1.0 + T24), 1.0 + T24 * (1 + 1e-9), 2.0 - T24, 0.1, -0.3, 1e-40,
                   -1e-45, 2.0**-149 * 0.5, 2.0**-126, 2.0**-126 * (1 - 2.0**-25), 2.0**-127 * 1.3, 1e-300, 3.4e38,
                   -3.4028234e38, 1.7e38, 123456.789])


def _split(x, q1, d, upper):
    u = (x - q1) / d
    i = (np.ceil(u) - 1 if upper else np.floor(u)).astype(np.int64)
    o = (u - i).astype(np.float32)
    if upper:
        o = np.where(o <= 0, np.float32(1e-7), o)
    else:
        o = np.where(o >= 1, np.float32(0.99999994), o)
    return i, o


@pytest.mark.parametrize("d", [(1.0, 1.0, 1.0), (0.5, 1.25, 0.7)])
def test_positions_and_velocities(d):
    cfg = config(0, cells=(20, 12, 8), ppc=11, seed=4)
    h = Hybrid(cfg, ni_max=cfg.n_particles + 7, coords=grd7(*cfg.nodes, *d))
    h.load_maxwellian()
    N = int(h.ni_tot[0])
    q1 = [q[0] for q in (h.coords.qx, h.coords.qy, h.coords.qz)]
    dd = [np.float64(np.float32(q[1] - q[0])) for q in (h.coords.qx, h.coords.qy, h.coords.qz)]
    rng = np.random.default_rng(8)
    frac = np.array([0.0, 1.0, 0.5, 1e-9, 1 - 1e-9, 1e-17, 1 - 1e-16, 0.25, 0.7])
    want = np.empty((N, 3))
    for m, upper in enumerate((True, False, True)):
        x = h.xp[:N, m].copy()
        i0, _ = _split(x, q1[m], dd[m], upper)
        y = q1[m] + (i0 + rng.choice(frac, N)) * dd[m]
        i1, _ = _split(y, q1[m], dd[m], upper)
        x = np.where(i1 == i0, y, x)  # the cells stay: the order does too
        h.xp[:N, m] = x
        i, o = _split(x, q1[m], dd[m], upper)
        want[:, m] = q1[m] + (i + o.astype(np.float64)) * dd[m]
        h.vp[:N, m] = rng.choice(SPEEDS, N)
        h.vp1[:N, m] = rng.choice(SPEEDS, N)
    v, v1 = h.vp[:N].copy(), h.vp1[:N].copy()
    h.mark_host_dirty()
    h.f32_begin()
    h.f32_end()
    h.sync_to_host()
    assert int(h.ni_tot[0]) == N
    assert np.max(np.abs(h.xp[:N] - want) / np.abs(want)) < 4 * 2.0**-52
    for got, had in ((h.vp, v), (h.vp1, v1)):
        ref = had.astype(np.float32).astype(np.float64)
        assert np.array_equal(got[:N], ref) and np.array_equal(np.signbit(got[:N]), np.signbit(ref))
    h.close()
