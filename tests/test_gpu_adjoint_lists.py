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


@pytest.mark.parametrize("bins,rmax,width,support", [(50, 4.0, 0.02, 6.0), (50, 4.0, 0.02, 30.0), (50, 4.0, 0.02, 40.0),
                                                     (512, 3.5, 0.015, 100.0)])
def test_wide_supports_of_the_bins_kernel(gpu, orc, bins, rmax, width, support):
    """A bin's kernel of its own value, however far away its row of bins begins: no weight is lost where the first
    bins' underflow."""
    cfg, u = _case(7, coul=True)
    _against_dual(orc, cfg, u, 6, 3, dict(gr_bins=bins, gr_every=2, gr_rmax=rmax, gr_width=width, gr_support=support))


def test_weights_of_one_pair(gpu):
    """g(r) of a single pair is a row of kernel values in 2^-32 steps, and the initial positions' gradient one term of
    them: no further off than the few roundings of a bin's own exponential."""
    from genesis_b200._lib import Handle
    cfg, _ = _case(8)
    L = cfg.size[0]
    bins, rmax, width, support = 512, 4.0, 0.1, 6.0
    d = 147.0 / 64.0  # exact through the wrap, as d - r is for centres in 256ths
    pos = np.array([[0.0, 0.0, 0.0], [d, 0.0, 0.0]])
    r = (np.arange(bins) + 0.5) * (rmax / bins)
    z = d - r
    c = L ** 3 / (4.0 * np.pi * r ** 2 * np.sqrt(2.0 * np.pi) * width)
    G = np.where(np.abs(z) < support * width, np.exp(-0.5 * (z / width) ** 2), 0.0)
    with Handle(cfg, "fp64") as h:
        h.set_state(pos, np.zeros_like(pos), np.zeros(2, np.uint8))  # at rest: the first drift leaves them in place
        _, g = h.adjoint_forward(1, checkpoint_every=1, gr_bins=bins, gr_rmax=rmax, gr_width=width, gr_support=support)
        assert np.max(np.abs(g / c - G)) <= 2.0 ** -33 * (1.0 + 2.0 ** -10)
        for k in np.flatnonzero(G)[::5]:
            w = np.zeros(bins)
            w[k] = 1.0
            _, _, (gx, _, _) = h.adjoint_backward(dl_dgr=w, initial_state=True)
            want = -c[k] * z[k] / width ** 2 * G[k]
            # three roundings of the exponent on each side, relative to it, and a dozen of the factors
            rel = 2.0 ** -50 * (4.0 + 0.5 * (z[k] / width) ** 2)
            assert abs(gx[1, 0] - want) <= rel * abs(want)


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_handles_of_different_bins_side_by_side(gpu, precision):
    """The many bins' launch after another handle's few: each handle as if it were alone."""
    from genesis_b200._lib import Handle
    cfg, u = _case(8)

    def forward(h, bins):
        h.set_universe(u)
        return h.adjoint_forward(6, checkpoint_every=2, gr_bins=bins, gr_rmax=4.5, gr_width=0.08)

    def backward(h, bins):
        return h.adjoint_backward(dl_dpotential=np.ones(6), dl_dgr=np.ones(bins))

    alone = []
    for bins in (512, 16):
        with Handle(cfg, precision) as h:
            alone.append((forward(h, bins), backward(h, bins)))
    with Handle(cfg, precision) as a, Handle(cfg, precision) as b:
        fa, fb = forward(a, 512), forward(b, 16)
        ba, bb = backward(a, 512), backward(b, 16)
        again = a.adjoint_forward(6, checkpoint_every=2, gr_bins=512, gr_rmax=4.5, gr_width=0.08)
    for (f, g), fwd, back in zip(alone, (fa, fb), (ba, bb)):
        for x, y in zip(f + g, fwd + back):
            assert np.array_equal(x, y)
    for x, y in zip(alone[0][0], again):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("n_side", [10, 11])  # 999 partners: lists sorted by ranges of slots; 1,330: cells every tick
def test_every_atom_within_the_cutoff_matches_dual_oracle(gpu, orc, n_side):
    cfg, u = _case(n_side, coul=True)
    cfg.coulomb_cutoff = 8.0
    _against_dual(orc, cfg, u, 3, 2, dict(gr_bins=30, gr_every=1, gr_rmax=6.0, gr_width=0.15, gr_support=6.0))


def _clump(n, radius, L=200.0):
    rng = np.random.default_rng(4)
    d = rng.normal(size=(n, 3))
    d *= (radius * rng.random(n) ** (1 / 3) / np.linalg.norm(d, axis=1))[:, None]
    return d + 0.25 * L, rng.integers(0, 10, n).astype(np.uint8)


@pytest.mark.parametrize("n,radius,slots", [(600, 2.0, 1), (3000, 4.0, 8), (20000, 3.0, 1)])
def test_clumps_for_any_checkpoint_spacing(gpu, n, radius, slots):
    """Rows, the pool beyond them (repeated calls, as it grows), and what no pool holds; slots of one residue in a
    clump.  The potential is the plain FP64 tick's, and the checkpoint spacing changes no bit."""
    from genesis_b200._lib import Handle
    cfg, _ = _case(8)
    cfg.size, cfg.dt = (200.0, 200.0, 200.0), 1e-7
    pos, elem = _clump(n, radius)
    if slots > 1:  # a clump's slots are those divisible by `slots`, the others spread over the box
        far = np.random.default_rng(5).uniform(-100.0, 100.0, size=(n * slots, 3))
        far[::slots] = pos
        pos, elem = far, np.repeat(elem, slots)
    T = 2
    with Handle(cfg, "fp64") as h:
        h.set_state(pos, np.zeros_like(pos), elem)
        want = h.step(T)["potential"]
    out = []
    for K in (1, 2):
        with Handle(cfg, "fp64") as h:
            h.set_state(pos, np.zeros_like(pos), elem)
            V, g = h.adjoint_forward(T, checkpoint_every=K, gr_bins=40, gr_rmax=3.0, gr_width=0.05)
            grad = h.adjoint_backward(dl_dpotential=np.ones(T), dl_dgr=np.ones(40), initial_state=True)
        assert np.max(np.abs(V - want) / np.abs(want)) <= 1e-10
        out.append((V, g, *grad[:2], *grad[2]))
    for a, b in zip(*out):
        assert np.array_equal(a, b)


def test_slots_eight_apart_cost_no_look_at_all_atoms(gpu):
    """A lattice whose neighbours' slots are eight apart against the same lattice in its own order: a lane that fell
    back to all 8,000 atoms took fifteen times as long."""
    import time
    from genesis_b200._lib import Handle
    cfg, u = _case(20)
    k = np.arange(u.n)
    best = []
    for order in (k, np.argsort((k % (u.n // 8)) * 8 + k // (u.n // 8))):
        with Handle(cfg, "mixed") as h:
            h.set_state(u.pos[order], u.vel[order], u.elem[order])
            took = []
            for _ in range(5):
                t = time.perf_counter()
                h.adjoint_forward(20, checkpoint_every=10)
                took.append(time.perf_counter() - t)
        best.append(min(took))
    assert best[1] <= 4.0 * best[0]


def test_more_cells_than_one_scan_of_tiles(gpu):
    """68,921 atoms on as many list cells: several scans in a row per tile, the last one ragged."""
    from genesis_b200._lib import Handle
    cfg, _ = _case(8)
    n, L = 41 ** 3, 41.5 * 1.2 * W.lattice_rc()
    cfg.size, cfg.dt = (L, L, L), 1e-7
    rng = np.random.default_rng(9)
    pos, elem = rng.uniform(-0.5 * L, 0.5 * L, size=(n, 3)), rng.integers(0, 10, n).astype(np.uint8)
    with Handle(cfg, "fp64") as h:
        h.set_state(pos, np.zeros_like(pos), elem)
        want = h.step(2)["potential"]
        h.set_state(pos, np.zeros_like(pos), elem)
        V, _ = h.adjoint_forward(2, checkpoint_every=1)
        gs, ge = h.adjoint_backward(dl_dpotential=np.array([0.0, 1.0]))
    assert np.max(np.abs(V - want) / np.abs(want)) <= 1e-10
    # V is linear in one factor on all epsilons but for the two ticks' drift at this step
    assert abs(ge @ np.asarray(cfg.epsilon_k) - V[1]) <= 1e-6 * abs(V[1])


@pytest.mark.parametrize("n_side,cutoff", [(10, 5.9), (11, 6.5)])  # two force cells an axis: lists of 860; cells
def test_wide_cutoffs_on_two_cells_match_dual_oracle(gpu, orc, n_side, cutoff):
    cfg, u = _case(n_side, coul=True)
    cfg.coulomb_cutoff = cutoff
    _against_dual(orc, cfg, u, 3, 2, dict(gr_bins=30, gr_every=1, gr_rmax=6.0, gr_width=0.15, gr_support=6.0))
