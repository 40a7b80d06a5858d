"""The mixed law through every pass that reads its pair table: isolated pairs
of ten kinds at distances across the core, the switch and the cutoff, the
same bits from each pass and within FP32's reach of the FP64 path."""
from __future__ import annotations

import numpy as np
import pytest

from genesis_b200 import elements as E
from genesis_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("coul,grav", [(False, False), (True, False), (True, True)])
def test_isolated_pairs(gpu, coul, grav):
    from genesis_b200._lib import Handle
    cfg = W.C1.config()
    n, step = 15, 16.0
    L = n * step
    cfg.size = (L, L, L)
    cfg.enable_electrostatics = coul
    cfg.enable_gravity, cfg.gravity_constant = grav, 0.01
    rng = np.random.default_rng(11)
    site = (np.stack(np.meshgrid(*[np.arange(n)] * 3, indexing="ij"), -1).reshape(-1, 3) + 0.5) * step - 0.5 * L
    d = rng.normal(size=site.shape)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    r = np.concatenate([rng.uniform(0.02, 1.2, 1000), rng.uniform(1.2, 5.1, 1000),
                        rng.uniform(5.1, 6.0, len(site) - 2000)])
    elem = rng.integers(0, 10, size=2 * len(site)).astype(np.uint8)
    zero = np.zeros((2 * len(site), 3))

    def acc(precision, dr=0.0, variant=None):
        with Handle(cfg, precision) as h:
            if variant is not None:
                h.set_kernel_variant(variant)
            h.set_state(np.concatenate([site, site + d * (r + dr)[:, None]]), zero, elem)
            if variant is None:
                h.forces()
            else:
                h.step(1, graph=False)  # from rest: the positions stay
            return h.get_state()[2]

    a = acc("fp64")
    # A displacement of FP32 cell-local coordinates (each end, the shift and the difference rounded at up to 8) is
    # within 2^-18 along the pair; across it, 2^-19 / r of the force.  Each of the law's few dozen FP32 operations is
    # within 2^-24 of terms whose cancellation the first part covers (they change by more than that over 2^-18), and
    # the sum is a multiple of 2^-32 over the mass.
    reach = sum(np.linalg.norm(acc("fp64", s * 2.0 ** -18) - a, axis=1) for s in (1, -1))
    size = np.linalg.norm(a, axis=1)
    mass = np.asarray(E.MASS)[elem]
    bound = 4 * reach + size * (2.0 ** -18 + 2.0 ** -18 / np.tile(r, 2)) + 2.0 ** -31 / mass
    first = None
    for variant in (1, 2, 3, 4, 5, 6, 7, 8, 0):
        got = acc("mixed", variant=variant)
        assert np.all(np.linalg.norm(got - a, axis=1) <= bound), variant
        if variant >= 5 or variant == 0:  # one frame of coordinates: the same bits
            first = got if first is None else first
            assert np.array_equal(got, first), variant


@pytest.mark.parametrize("n_side", [3, 4, 20, 21, 27, 28, 35, 36, 50, 51])
def test_lanes_of_the_per_tick_pass(gpu, n_side):
    """The per-tick pass with 16, 8, 4, 2 and 1 lanes per atom (sizes on both
    sides of each line, grids of one to three cells too) against one thread
    per atom: the same integer sums."""
    from genesis_b200._lib import Handle
    wl = W.Workload("lanes", n_side=n_side, temperature=200.0, steps=10, electrostatics=True)
    cfg, u = wl.config(), wl.generate()
    out = []
    for variant in (1, 0):
        with Handle(cfg, "mixed") as h:
            h.set_universe(u)
            h.set_kernel_variant(variant)
            h.half_kick()
            h.drift()
            h.wrap()
            out.append((h.forces(), h.get_state()))
    assert out[0][0] == out[1][0]
    for a, b in zip(out[0][1], out[1][1]):
        assert np.array_equal(a, b)
