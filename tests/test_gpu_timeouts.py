"""Launches whose grid barrier gives up: the status, the launches queued behind
them, and the handle afterwards.  A limit of no polls makes every wait run out
at once; nothing waits for long and nothing faults."""
from __future__ import annotations

import numpy as np
import pytest

from genesis_b200 import workloads as W

pytestmark = pytest.mark.gpu

TIMEOUT, STATE = -7, -9
POLLS = 1 << 22


def _handle(precision="mixed"):
    from genesis_b200._lib import Handle
    wl = W.C1.scaled(9)
    return Handle(wl.config(), precision), wl.generate()


def _status(call):
    from genesis_b200._lib import GxError
    with pytest.raises(GxError) as e:
        call()
    return e.value.status


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_timed_out_ticks_lose_the_state_and_no_more(gpu, precision):
    ref, u = _handle(precision)
    with ref:
        ref.set_universe(u)
        want = ref.step(300, graph=True), ref.get_state()
    h, _ = _handle(precision)
    with h:
        h.set_universe(u)
        h.step(3, graph=True)
        h.set_wait_polls(0)
        assert _status(lambda: h.step(600, stats=False, graph=True)) == TIMEOUT  # its second and third launch find the word set
        for call in (lambda: h.step(1, graph=True), h.get_state, h.forces, h.stats, h.snapshot_world, lambda: h.xyz_frame(0),
                     lambda: h.clusters(), lambda: h.adjoint_forward(1)):
            assert _status(call) == STATE
        h.set_universe(u)
        h.set_wait_polls(POLLS)
        got = h.step(300, graph=True), h.get_state()
        for f in want[0].dtype.names:
            assert np.array_equal(want[0][f], got[0][f])
        for x, y in zip(want[1], got[1]):
            assert np.array_equal(x, y)


def test_queued_steps_behind_a_timeout(gpu):
    h, u = _handle()
    with h:
        h.set_universe(u)
        h.set_step_async(True)
        h.set_wait_polls(0)
        h.step(2, stats=False, graph=True)
        h.set_wait_polls(POLLS)
        h.step(600, stats=False, graph=True)  # queued before the error is known: does nothing
        assert _status(h.synchronize) == TIMEOUT
        assert _status(h.get_state) == STATE
        # a state uploaded while the error is still queued stands
        h.set_universe(u)
        h.set_wait_polls(0)
        h.step(2, stats=False, graph=True)
        h.set_wait_polls(POLLS)
        h.set_universe(u)
        assert _status(h.synchronize) == TIMEOUT
        pos, vel, _ = h.get_state()
        assert np.array_equal(pos, u.pos) and np.array_equal(vel, u.vel)
        h.step(5, stats=False, graph=True)
        h.synchronize()
        got = h.get_state()
    ref, _ = _handle()
    with ref:
        ref.set_universe(u)
        ref.step(5, graph=True)
        for x, y in zip(ref.get_state(), got):
            assert np.array_equal(x, y)


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_timed_out_adjoint(gpu, precision):
    spec = dict(checkpoint_every=100, gr_bins=20, gr_rmax=4.0, gr_width=0.1)
    h, u = _handle(precision)
    with h:
        h.set_universe(u)
        V, g = h.adjoint_forward(300, **spec)
        want = h.adjoint_backward(dl_dpotential=np.ones(300), dl_dgr=np.ones(20))
        h.set_wait_polls(0)
        assert _status(lambda: h.adjoint_backward(dl_dpotential=np.ones(300))) == TIMEOUT
        h.set_wait_polls(POLLS)
        got = h.adjoint_backward(dl_dpotential=np.ones(300), dl_dgr=np.ones(20))  # the checkpoints stand
        for x, y in zip(want, got):
            assert np.array_equal(x, y)
        h.set_wait_polls(0)
        assert _status(lambda: h.adjoint_forward(300, **spec)) == TIMEOUT
        assert _status(lambda: h.adjoint_backward(dl_dpotential=np.ones(300))) == STATE
        h.set_wait_polls(POLLS)
        V2, g2 = h.adjoint_forward(300, **spec)
        assert np.array_equal(V, V2) and np.array_equal(g, g2)
        for x, y in zip((u.pos, u.vel), h.get_state()):
            assert np.array_equal(x, y)
