"""FP32 runs of two contexts on one GPU, each in its own host thread, on a grid
whose field step is one cooperative launch (above the cluster form's 4096 nodes
and below FIELD_LOOP_NODES): the launches take turns on the device, so each run
gives the bits it gives alone."""
import threading

import numpy as np
import pytest

from helpers import make_hybrid

pytestmark = pytest.mark.gpu
KW = dict(cells=(24, 20, 16), ppc=6, db=0.03)  # 7680 nodes


def _make(seed):
    h = make_hybrid(seed=seed, **KW)
    h.f32_begin()
    return h


def _end(h):
    h.f32_end()
    h.sync_to_host()
    return {n: getattr(h, n).copy() for n in ("xp", "vp", "b1", "b12", "np", "up", "E")}


def test_two_threads_give_the_bits_of_one():
    want = []
    for seed in (5, 6):
        h = _make(seed)
        h.f32_run(24)
        want.append(_end(h))
        h.close()
    hs = [_make(5), _make(6)]
    errs, gate = [None, None], threading.Barrier(2, timeout=60)

    def work(r):
        try:
            gate.wait()
            for n in (8, 1, 15):
                hs[r].f32_run(n)
        except Exception as e:  # reported below
            errs[r] = e

    th = [threading.Thread(target=work, args=(r,)) for r in range(2)]
    for t in th:
        t.start()
    for t in th:
        t.join(timeout=300)
    assert not any(t.is_alive() for t in th) and errs == [None, None], errs
    for h, w in zip(hs, want):
        got = _end(h)
        for n in w:
            assert np.array_equal(got[n], w[n]), n
        h.close()
