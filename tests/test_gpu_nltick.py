"""The one-launch ticks of small universes (automatic variant, captured or
one-launch step) against the per-kernel ticks of the same handle settings
(eager step): the same sums in the same order, so the same bits."""
from __future__ import annotations

import numpy as np
import pytest

from genesis_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _pair(cfg, u, ticks, bonds=None, skin=None, precision="mixed"):
    from genesis_b200._lib import Handle
    out = []
    for graph in (True, False):
        h = Handle(cfg, precision)
        h.set_universe(u)
        if bonds is not None:
            h.set_bonds(bonds)
        if skin is not None:
            h.set_list_skin(skin)
        l0 = h.launches
        st = [h.step(k, stats=rec, graph=graph) for k, rec in ticks]
        out.append((st, h.get_state(), h.list_rebuilds(), h.stats(), h.launches - l0))
        h.close()
    (sa, xa, ra, ka, la), (sb, xb, rb, kb, lb) = out
    assert la < lb  # the two paths are not the same one
    assert ra == rb
    assert ka == kb
    for a, b in zip(xa, xb):
        assert np.array_equal(a, b)
    for a, b in zip(sa, sb):
        assert (a is None) == (b is None) and (a is None or np.array_equal(a, b))
    return ra


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("n_side,coul,target", [(8, False, 0.0), (9, True, 40.0), (16, False, 0.0), (16, True, 40.0),
                                                (25, True, 0.0), (40, True, 300.0)])
def test_one_launch_ticks_match_the_per_kernel_ticks(gpu, n_side, coul, target, precision):
    wl = W.Workload("tick check", n_side=n_side, temperature=200.0, steps=10, electrostatics=coul,
                    thermostat=target > 0.0, thermostat_temperature=target if target > 0.0 else 300.0)
    rebuilds = _pair(wl.config(), wl.generate(), [(1, True), (2, False), (7, True), (1, False), (9, True)],
                     precision=precision)
    assert rebuilds >= 2


def test_one_launch_gravity_and_no_walls(gpu):
    wl = W.Workload("tick check", n_side=11, temperature=100.0, steps=10, electrostatics=True)
    cfg = wl.config()
    cfg.enable_gravity, cfg.gravity_constant = True, 1e-3
    _pair(cfg, wl.generate(), [(6, True), (3, False)])
    cfg.enable_boundaries = False
    _pair(cfg, wl.generate(), [(6, True), (3, False)])


def test_one_launch_spring_and_zero_skin(gpu):
    wl = W.C2.scaled(10)
    cfg, u = wl.config(), wl.generate()
    i = np.arange(0, u.n - 1, 2, dtype=np.uint32)
    bonds = np.stack([i, i + 1], 1)  # neighbours along the lattice's fastest axis
    _pair(cfg, u, [(5, True), (4, False)], bonds=bonds)
    assert _pair(cfg, u, [(3, True), (3, False)], skin=0.0) >= 5


def test_one_launch_sparse_box_and_overflowing_clump(gpu):
    # more list cells than one scan tile, and atoms whose lists overflow
    wl = W.Workload("tick check", n_side=10, temperature=20.0, steps=10)
    cfg, u = wl.config(), wl.generate()
    L = 110.0
    cfg.size = (L, L, L)
    u.box[:] = L
    rng = np.random.default_rng(3)
    u.pos[:300] = rng.normal(scale=2.5, size=(300, 3))
    u.pos[300:] = rng.uniform(-0.5 * L, 0.5 * L, size=(700, 3))
    u.vel[:] *= 0.01
    _pair(cfg, u, [(3, True), (1, False)])
    _pair(cfg, u, [(3, True), (1, False)], precision="fp64")


def test_one_launch_tick_reports_and_recovers_from_a_non_finite_velocity(gpu):
    from genesis_b200._lib import GxError, Handle
    wl = W.C1.scaled(9)
    cfg, u = wl.config(), wl.generate()
    bad = u.vel.copy()
    bad[5, 1] = np.nan
    with Handle(cfg, "mixed") as h:
        h.set_universe(u)
        h.step(2, graph=True)
        h.set_dynamic(u.pos, bad, np.zeros_like(u.pos))
        with pytest.raises(GxError):
            h.step(2, graph=True)
        h.set_dynamic(u.pos, u.vel, np.zeros_like(u.pos))
        st = h.step(3, graph=True)
    with Handle(cfg, "mixed") as h:
        h.set_universe(u)
        want = h.step(3, graph=True)
    assert np.array_equal(st["potential"], want["potential"])


def test_autotuned_variant_is_the_same_tick_on_another_handle(gpu):
    """A small universe's autotuner keeps the one-launch tick, and the variant it reports gives it elsewhere."""
    from genesis_b200._lib import Handle
    wl = W.Workload("tick check", n_side=8, temperature=100.0, steps=10)
    cfg, u = wl.config(), wl.generate()
    out = []
    with Handle(cfg, "mixed") as a, Handle(cfg, "mixed") as b:
        for h in (a, b):
            h.set_universe(u)
        best, _ = a.autotune(reps=20)
        b.set_kernel_variant(best)
        b.set_list_skin(a.list_config()[0])
        for h in (a, b):
            h.step(1, graph=True)
            l0 = h.launches
            h.step(20, graph=True)
            out.append(h.launches - l0)
    assert out == [2, 2]  # the ticks, and the words read back


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("target", [0.0, 150.0])
def test_ticks_across_launches(gpu, precision, target):
    """Calls of more ticks than one launch takes (256): the records' places, the pending scale, the frame's parity."""
    wl = W.Workload("tick check", n_side=8, temperature=200.0, steps=10, thermostat=target > 0.0,
                    thermostat_temperature=target if target > 0.0 else 300.0)
    _pair(wl.config(), wl.generate(), [(257, True), (513, True), (258, False), (3, True)], precision=precision)


@pytest.mark.parametrize("precision,n_side,one", [("mixed", 8, True), ("mixed", 40, True), ("mixed", 41, False),
                                                  ("fp64", 8, True), ("fp64", 29, True), ("fp64", 30, False)])
def test_sizes_that_run_in_one_launch(gpu, precision, n_side, one):
    """The exact launches of a call on both sides of each limit: one per 256 ticks and the read-back's."""
    from genesis_b200._lib import Handle
    wl = W.Workload("tick check", n_side=n_side, temperature=100.0, steps=10)
    with Handle(wl.config(), precision) as h:
        h.set_universe(wl.generate())
        h.step(1, graph=True)
        for ticks in (5,) if n_side > 8 else (1, 5, 256, 257, 513):
            l0 = h.launches
            h.step(ticks, graph=True)
            assert (h.launches - l0 == -(-ticks // 256) + 1) == one
        if precision == "mixed" and one:  # a work shape is the per-kernel tick's, as is any other variant
            l0 = h.launches
            h.set_kernel_variant(5)
            h.step(5, graph=True)
            assert h.launches - l0 > 2
            h.set_kernel_variant(6)
            h.set_list_threads(4)
            l0 = h.launches
            h.step(5, graph=True)
            assert h.launches - l0 > 2


def test_the_default_block_is_no_shape(gpu):
    """Far ends in global memory is the default: setting it, or going back to it, keeps the one-launch tick."""
    from genesis_b200._lib import Handle
    wl = W.Workload("tick check", n_side=8, temperature=100.0, steps=10)
    with Handle(wl.config(), "mixed") as h:
        h.set_universe(wl.generate())
        for block, one in ((0, True), (128, False), (0, True)):
            h.set_list_block(block)
            h.step(1, graph=True)
            l0 = h.launches
            h.step(5, graph=True)
            assert (h.launches - l0 == 2) == one
