"""The FP32-prefiltered g(r) pass (grids of at least 3 cells per axis, at most
1,024 bins) against the oracle's exact counts and against the general FP64
pass, which more bins select: 2,048 bins of half, a quarter ... the width
add up to exactly the same counts (d / dr scales by a power of two)."""
from __future__ import annotations

import numpy as np
import pytest

from genesis_b200 import synth
from genesis_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _handle(pos, box, elem=None):
    from genesis_b200._lib import Handle
    cfg = W.C1.config()
    cfg.size = tuple(box)
    h = Handle(cfg, "fp64")
    h.set_state(pos, np.zeros_like(pos), np.zeros(len(pos), np.uint8) if elem is None else elem)
    return h


def _grouped(h, r_max, nbins, **kw):
    fine = h.radial_distribution(r_max, 2048, 0, **kw)[0]
    return fine.reshape(nbins, -1).sum(1)


@pytest.mark.parametrize("nbins", [1, 7, 16, 256, 1024])
def test_distances_on_bin_edges(gpu, orc, nbins):
    # a perfect unit lattice: every distance is a root of an integer, most of them on edges
    n = 16
    pos = np.stack(np.meshgrid(*[np.arange(n) - 7.5] * 3, indexing="ij"), -1).reshape(-1, 3).copy()
    h = _handle(pos, (n, n, n))
    counts, bins, _, _ = h.radial_distribution(4.0, nbins)
    want, b, _, _, rc = orc.radial_distribution(pos, (n, n, n), 4.0, nbins)
    assert rc == 0 and np.array_equal(counts, want) and np.array_equal(bins, b)


@pytest.mark.parametrize("nbins", [1, 255, 1024])
def test_uneven_box_clumps_and_coincident_atoms(gpu, orc, nbins):
    box = (30.0, 47.0, 61.0)
    rng = np.random.default_rng(5)
    u = synth.uniform_box(5000, box, seed=2)
    pos = u.pos.copy()
    pos[:700] = rng.normal(scale=1.0, size=(700, 3)) + np.array([14.0, -20.0, 30.0])
    pos[700:720] = pos[720:740]  # distance zero
    pos[740:760] = pos[760:780] + 1e-17
    pos = (pos + 0.5 * np.array(box)) % np.array(box) - 0.5 * np.array(box)
    h = _handle(pos, box, u.elem)
    for between in (None, (2, 2), (0, 6)):
        counts, _, _, _ = h.radial_distribution(9.9, nbins, between=between)
        want, _, _, _, rc = orc.radial_distribution(pos, box, 9.9, nbins, elem=u.elem, between=between)
        assert rc == 0 and np.array_equal(counts, want)


@pytest.mark.parametrize("n_side,r_max", [(20, 17.25), (41, 9.0), (45, 17.25)])
def test_whole_state_matches_the_general_pass(gpu, n_side, r_max):
    # 8,000 atoms two at a time per warp, 68,921 and 91,125 eight at a time
    u = synth.lattice(n_side, 2.76, 0.15, 60.0, 0.01, seed=4)
    h = _handle(u.pos, u.box, u.elem)
    for nbins in (1, 256, 1024):
        assert np.array_equal(h.radial_distribution(r_max, nbins, 0)[0], _grouped(h, r_max, nbins))
    assert np.array_equal(h.radial_distribution(r_max, 256, 0, between=(3, 7))[0],
                          _grouped(h, r_max, 256, between=(3, 7)))


def test_atoms_outside_the_box(gpu):
    u = synth.lattice(20, 2.76, 0.15, 60.0, 0.01, seed=4)
    rng = np.random.default_rng(0)
    pos = u.pos + u.box * rng.integers(-3, 4, size=(u.n, 3))
    pos[::50] += u.box * 1e7  # where the FP64 differences themselves round
    h = _handle(pos, u.box, u.elem)
    assert np.array_equal(h.radial_distribution(17.25, 256, 0)[0], _grouped(h, 17.25, 256))
