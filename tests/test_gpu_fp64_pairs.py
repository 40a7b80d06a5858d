"""The FP64 law bit for bit: thousands of isolated pairs at distances across
the core, the switch and the cutoff, so that an acceleration is one pair's
force over a mass, against the oracle's exact arithmetic, through the
per-tick pass (gx_forces) and the list pass (gx_step)."""
from __future__ import annotations

import numpy as np
import pytest

from genesis_b200 import elements as E
from genesis_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _pairs(seed, coul, grav, coulomb_cutoff):
    cfg = W.C1.config()
    n, step = 15, 16.0
    L = n * step
    cfg.size = (L, L, L)
    cfg.enable_electrostatics, cfg.coulomb_cutoff = coul, coulomb_cutoff
    cfg.enable_gravity, cfg.gravity_constant = grav, 0.01
    rng = np.random.default_rng(seed)
    site = (np.stack(np.meshgrid(*[np.arange(n)] * 3, indexing="ij"), -1).reshape(-1, 3) + 0.5) * step - 0.5 * L
    d = rng.normal(size=site.shape)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    r = np.concatenate([rng.uniform(0.02, 1.2, 1000), rng.uniform(1.2, 5.1, 1000),
                        rng.uniform(5.1, 7.0, len(site) - 2000)])
    pos = np.concatenate([site, site + d * r[:, None]])
    elem = rng.integers(0, 10, size=len(pos)).astype(np.uint8)
    charge = np.where(rng.random(len(pos)) < 0.4, 0.0, rng.normal(size=len(pos)) * 10.0 ** rng.integers(-3, 3, len(pos)))
    mass = np.asarray(E.MASS)[elem] * rng.uniform(0.5, 2.0, size=len(pos))
    return cfg, np.ascontiguousarray(pos), elem, charge, mass


def _partners(pos, L, reach):
    """Atoms within reach of each atom."""
    out = np.zeros(len(pos), dtype=int)
    for k in range(0, len(pos), 250):
        d = pos[k:k + 250, None] - pos[None]
        d -= L * np.round(d / L)
        out[k:k + 250] = ((d * d).sum(-1) < reach * reach).sum(1) - 1
    return out


@pytest.mark.parametrize("coul,grav,cutoff", [(False, False, 2.5), (True, False, 2.5), (True, True, 2.8)])
def test_isolated_pairs_are_bit_exact(gpu, orc, coul, grav, cutoff):
    from genesis_b200._lib import Handle
    cfg, pos, elem, charge, mass = _pairs(7, coul, grav, cutoff)
    zero = np.zeros_like(pos)
    with Handle(cfg, "fp64") as h:
        h.set_state(pos, zero, elem, charge=charge, mass=mass)
        h.forces()
        acc = h.get_state()[2]
        want = orc.forces(cfg, pos, elem, charge, mass)
        # where two pairs reach the same atom (the longest ones) the order of their sum is free
        lone = _partners(pos, cfg.size[0], 7.0) <= 1
        assert lone.sum() > 6000
        # gravity's strength is (G m_a) m_b in the reference's pair (a, b) and (G m_i) m_j for atom i here: the two
        # products differ by two roundings, so by 2^-52 of that term, and the sum with the others by one more
        bound = np.zeros(len(pos))
        if grav:
            cfg.enable_gravity = False
            rest = orc.forces(cfg, pos, elem, charge, mass)[0]
            cfg.enable_gravity = True
            size = lambda a: np.linalg.norm(a, axis=1)  # noqa: E731
            bound = 2.0 ** -50 * (size(want[0] - rest) + size(want[0]))

        def same(a, b, scale=1.0):
            return bool(np.all(np.linalg.norm(a - b, axis=1)[lone] <= scale * bound[lone]))

        assert same(acc, want[0])
        h.set_state(pos, zero, elem, charge=charge, mass=mass)
        h.step(1)
        got = h.get_state()
        ref = orc.ticks(cfg, pos, zero, zero, elem, charge, mass, 1)
        assert np.array_equal(got[0], ref[0])  # drifted from rest
        assert same(got[2], ref[2]) and same(got[1], ref[1], cfg.dt)
