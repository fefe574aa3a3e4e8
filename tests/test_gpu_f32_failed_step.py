"""A step of the FP32 form that fails after its sort, on grids where a run of
several steps leaves the sorted moves to the next pass 1: the state is then the
one that single steps, which move the ions themselves, leave behind -- when the
inflow outgrows the arrays, and when the exchange of the last moments fails."""
import numpy as np
import pytest

from swap_gb300 import abi
from swap_gb300.hybrid import Hybrid, config

pytestmark = pytest.mark.gpu
CELLS = (64, 60, 40)  # 153600 cells, above FIELD_LOOP_NODES
ECAPACITY, EEXCHANGE = 4, 9


def _make(room):
    cfg = config(1, cells=CELLS, ppc=4, seed=12)
    cfg.sources.update(inflow_ppc=40)  # ten times what leaves
    h = Hybrid(cfg, ni_max=cfg.n_particles + room, work_arrays=False)
    h.load_maxwellian()
    h.set_sources(cfg.make_sources())
    h.mark_host_dirty()
    h.f32_begin()
    return h


def _run_until_it_fails(h, n, each):
    for _ in range(n // each):
        h.f32_run(each)


def _same_end(a, b):
    assert a.f32_count() == b.f32_count()
    for h in (a, b):
        h.f32_end()
        h.sync_to_host()
    N = int(a.ni_tot[0])
    assert N == int(b.ni_tot[0]) > a.cfg.n_particles
    for n in ("xp", "vp", "vp1", "mrat", "beta_p"):
        assert np.array_equal(getattr(a, n)[:N], getattr(b, n)[:N]), n
    # every ion inside: none of an older order's places
    for m, q in enumerate((a.coords.qx, a.coords.qy, a.coords.qz)):
        assert (a.xp[:N, m] >= q[0]).all() and (a.xp[:N, m] <= q[-2]).all()
    for n in ("b1", "b12", "np", "up", "E", "aj"):
        assert np.array_equal(getattr(a, n), getattr(b, n)), n


def test_inflow_beyond_the_room():
    a, b = _make(30000), _make(30000)
    for h, each in ((a, 8), (b, 1)):
        with pytest.raises(abi.SwapError) as e:
            _run_until_it_fails(h, 8, each)
        assert e.value.code == ECAPACITY
        assert h.f32_count() == h.ni_max
        with pytest.raises(abi.SwapError) as e:  # start[] counts ions that there is no room for
            h.f32_run(1)
        assert e.value.code == ECAPACITY
    _same_end(a, b)
    a.close()
    b.close()


def test_exchange_that_fails_after_the_sort():
    a, b = _make(200000), _make(200000)
    for h, each in ((a, 6), (b, 1)):
        calls = []
        # three exchanges a step; the last of the third step comes after its sort was queued
        h.set_exchange(lambda data, count, kind, stream: calls.append(0) or (5 if len(calls) == 9 else 0))
        with pytest.raises(abi.SwapError) as e:
            _run_until_it_fails(h, 6, each)
        assert e.value.code == EEXCHANGE and len(calls) == 9
        h.f32_run(2)  # the state stays usable
    _same_end(a, b)
    a.close()
    b.close()
