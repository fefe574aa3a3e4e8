"""The FP64 cell search (get_interp_weights, gutsp.f:1396-1404) at positions
where its index arithmetic can go wrong, against numpy's comparisons."""
import numpy as np
import pytest

from swap_gb300 import abi
from swap_gb300.grid import grd7
from swap_gb300.hybrid import Hybrid, config

pytestmark = pytest.mark.gpu

FAR = (np.inf, -np.inf, 1e300, -1e300, 3.5e38, 1e12, 4294967301.0, 2147483649.0, 2147483647.5, -2147483649.5, np.nan)


def _make(cells=(7, 5, 6), ppc=4, coords=None):
    cfg = config(0, cells=cells, ppc=ppc, seed=2)
    h = Hybrid(cfg, coords=coords)
    h.load_maxwellian()
    h.mark_host_dirty()
    return h


@pytest.mark.parametrize("axis", [0, 1, 2])
def test_positions_far_outside_are_reported(axis):
    h = _make()
    keep = h.xp.copy(order="F")
    for bad in FAR:
        h.xp[11, axis] = bad
        h.mark_host_dirty(h.xp)
        with pytest.raises(abi.SwapError, match="EDOMAIN"):
            h.get_interp_weights(h.xp)
        h.xp[...] = keep
        h.mark_host_dirty(h.xp)
        h.get_interp_weights(h.xp)
    h.close()


def _minus_zero_nodes(nodes, at):
    """Unit spacings with node `at` (1-based) of x and z at -0.0."""
    co = grd7(*nodes)
    for q, n in ((co.qx, nodes[0]), (co.qz, nodes[2])):
        q[...] = -(at - 1.0 - np.arange(n))
        assert q[at - 1] == 0.0 and np.signbit(q[at - 1])
    return co


@pytest.mark.parametrize("at", [1, 4])
def test_a_node_at_minus_zero(at):
    cells = (7, 5, 6)
    co = _minus_zero_nodes(tuple(c + 2 for c in cells), at)
    h = _make(cells, coords=co)
    n = int(h.ni_tot[0])
    tiny = 5e-324
    picks = np.array([0.0, -0.0, tiny, -tiny, 0.5, -0.5, 1.0, 2.0])
    rng = np.random.default_rng(1)
    for m, q in ((0, co.qx), (2, co.qz)):
        x = rng.choice(picks if at > 1 else picks[[2, 4, 6, 7]], n)
        h.xp[:n, m] = x
        # q(i) < x <= q(i+1), gutsp.f:1396-1401
        want = np.array([int(np.nonzero((q[:-1] < v) & (v <= q[1:]))[0][0]) + 1 for v in x])
        h.mark_host_dirty()
        h.get_interp_weights(h.xp)
        h.sync_to_host(h.ijkp)
        assert np.array_equal(h.ijkp[:n, m], want)
    if at == 1:  # +0 is not above the first node
        h.xp[7, 0] = 0.0
        h.mark_host_dirty(h.xp)
        with pytest.raises(abi.SwapError, match="EDOMAIN"):
            h.get_interp_weights(h.xp)
    h.close()


def test_a_move_onto_a_face_at_minus_zero():
    """x = +0 at the first node -0.0 wraps to the far face (gutsp.f:490-498), in the passes as in the operators."""
    cells = (7, 5, 6)
    co = _minus_zero_nodes(tuple(c + 2 for c in cells), 1)
    cfg = config(0, cells=cells, ppc=4, seed=2, dt=0.5, ntsub=4, u=(0.0, 0.0, 0.0), vth=1e-30)
    got = []
    for det in (False, True):  # the passes; the deterministic form: operators
        h = Hybrid(cfg, coords=co)
        h.load_maxwellian()
        n = int(h.ni_tot[0])
        h.vp[:n] = h.vp1[:n] = 0.0
        h.b1[...] = h.b12[...] = h.b1p2[...] = h.bt[...] = h.b0
        h.xp[3] = (0.25, 2.5, 0.25)
        h.vp[3] = h.vp1[3] = (-1.0, 0.0, -1.0)
        h.b0[...] = 0.0
        for b in (h.b1, h.b12, h.b1p2, h.bt):  # no field: the ion goes straight, by 0.25 to exactly zero
            b[...] = 0.0
        h.mark_host_dirty()
        h.set_deterministic(det)
        h._check(h.lib.swap_ion_step_pre(h.ctx))
        h.sync_to_host()
        got.append(h.xp[3].copy())
        h.close()
    assert np.array_equal(got[0], got[1]) and got[0][0] == 7.0 and got[0][2] == 6.0


def test_a_refused_call_leaves_the_cells_of_the_one_before():
    h = _make()
    n = int(h.ni_tot[0])
    h.get_interp_weights(h.xp)
    h.sync_to_host(h.ijkp)
    had = h.ijkp[:n].copy()
    h.get_interp_weights(h.xp)  # current on the device alone
    keep = h.xp.copy(order="F")
    h.xp[:n] = h.xp[:n][::-1].copy()
    h.xp[n // 2, 2] = 1e9
    h.mark_host_dirty(h.xp)
    with pytest.raises(abi.SwapError, match="EDOMAIN"):
        h.get_interp_weights(h.xp)
    h.sync_to_host(h.ijkp)
    assert np.array_equal(h.ijkp[:n], had)
    h.xp[:n] = keep[:n][::-1].copy()
    h.mark_host_dirty(h.xp)
    h.get_interp_weights(h.xp)
    h.sync_to_host(h.ijkp)
    assert np.array_equal(h.ijkp[:n], had[::-1])
    h.close()
