"""The adjoint's lists in the one-launch ticks: axes of one and two force
cells (a pair counts as often as in the reference's pair list), a clump whose
lists overflow, more bins than a static histogram holds, a horizon longer
than one launch, and every atom alone.  Same bounds as test_gpu_adjoint."""
from __future__ import annotations

import dataclasses

import numpy as np
import pytest

from genesis_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _case(n_side, coul=False, temperature=60.0):
    wl = W.Workload("adjoint lists", n_side=n_side, temperature=temperature, steps=1, seed=5, electrostatics=coul)
    return wl.config(), wl.generate()


def _close(a, b, rel, floor):
    a, b = np.asarray(a), np.asarray(b)
    return bool(np.all(np.abs(a - b) <= rel * np.abs(b) + floor * np.abs(b).max()))


def _against_dual(orc, cfg, u, T, K, gr):
    from genesis_b200._lib import Handle
    with Handle(cfg, "fp64") as h:
        h.set_universe(u)
        V, g = h.adjoint_forward(T, checkpoint_every=K, **gr)
        dV, dg = np.linspace(0.5, 1.5, T), np.cos(np.arange(len(g)))
        gs, ge = h.adjoint_backward(dl_dpotential=dV, dl_dgr=dg)
    Vo, go, dVo, dgo = orc.adjoint_forward(cfg, u.pos, u.vel, np.zeros_like(u.pos), u.elem, u.charge, u.mass, T,
                                           nthreads=4, dual=True, **gr)
    want = dV @ dVo + dg @ dgo
    assert np.max(np.abs(V - Vo) / np.abs(Vo)) <= 1e-10
    assert np.max(np.abs(g - go)) <= 1e-9 * np.max(np.abs(go))
    assert _close(np.concatenate([gs, ge]), want, 1e-7, 1e-9)


@pytest.mark.parametrize("n_side,coul", [(4, False), (5, True), (6, False)])
def test_small_boxes_match_dual_oracle(gpu, orc, n_side, coul):
    cfg, u = _case(n_side, coul)  # 1, 2 and 2 force cells per axis
    _against_dual(orc, cfg, u, 12, 5, dict(gr_bins=30, gr_every=3, gr_rmax=4.5, gr_width=0.15, gr_support=6.0))


def test_two_cells_along_one_axis(gpu, orc):
    cfg, u = _case(6)
    size = np.array([16.56, 22.08, 30.0])
    cfg.size = tuple(size)
    u.box[:] = size
    _against_dual(orc, cfg, u, 8, 3, dict(gr_bins=30, gr_every=1, gr_rmax=4.5, gr_width=0.15, gr_support=6.0))


def test_overflowing_lists_match_dual_oracle(gpu, orc):
    cfg, u = _case(8)
    L = 40.0
    cfg.size, cfg.dt = (L, L, L), 1e-3
    u.box[:] = L
    side = np.arange(7) * 0.9 - 2.7
    clump = np.stack(np.meshgrid(side, side, side, indexing="ij"), -1).reshape(-1, 3)
    rng = np.random.default_rng(1)
    pos = rng.uniform(-0.5 * L, 0.5 * L, size=(u.n, 3))
    pos[:343] = clump + rng.normal(scale=0.02, size=clump.shape)
    pos[343:] += np.where(np.linalg.norm(pos[343:], axis=1) < 8.0, 12.0, 0.0)[:, None]
    u = dataclasses.replace(u, pos=(pos + 0.5 * L) % L - 0.5 * L)
    _against_dual(orc, cfg, u, 4, 3, dict(gr_bins=30, gr_every=2, gr_rmax=4.5, gr_width=0.15, gr_support=6.0))


def test_many_bins_long_horizon_and_far_atoms(gpu):
    from genesis_b200._lib import Handle
    cfg, u = _case(8, temperature=30.0)
    out = []
    for K in (20, 300):
        with Handle(cfg, "mixed") as h:
            h.set_universe(u)
            V, g = h.adjoint_forward(270, checkpoint_every=K, gr_bins=512, gr_every=7, gr_rmax=4.8, gr_width=0.1)
            out.append((V, g, *h.adjoint_backward(dl_dpotential=np.ones(270), dl_dgr=np.ones(512))))
    for a, b in zip(*out):
        assert np.array_equal(a, b)
    cfg.size = (500.0, 500.0, 500.0)  # no atom within reach of another, more list cells than one scan tile
    far = np.stack(np.meshgrid(*[np.arange(8) * 60.0 - 210.0] * 3, indexing="ij"), -1).reshape(-1, 3)
    with Handle(cfg, "fp64") as h:
        h.set_state(far, np.zeros_like(far), u.elem)
        V, g = h.adjoint_forward(3, checkpoint_every=2, gr_bins=16, gr_rmax=4.8, gr_width=0.1)
        gs, ge = h.adjoint_backward(dl_dpotential=np.ones(3), dl_dgr=np.ones(16))
    assert not V.any() and not g.any() and not gs.any() and not ge.any()
