"""The calls a user of this library makes, as measurable cases.

A case is a dict of plain values; `listed` names twelve, `draw` gives more of
the same ranges.  Universes come from `genesis_b200.workloads` and
`genesis_b200.synth` (cubic lattices of side `n`, the ten elements or Na/O),
with the handle's default settings unless a case says otherwise.

Kinds:

* ``run``       a trajectory segment: `ticks` recorded ticks replayed from
                CUDA graphs, optionally one g(r) at its end (the reference's
                8,192-atom subsample), and the state copied out
* ``host_tick`` one tick against the host's own columns (a drop-in system)
* ``observed``  ticks with the bond observation after each, its bonds feeding
                the spring of the next tick
* ``schedule``  the reference's schedule, system by system (`GpuUniverse`)
* ``sweep``     a temperature sweep of many uneven replicas as one batch
* ``adjoint``   a trajectory and its gradients for two losses
* ``lens``      structure analysis of one state: friends-of-friends and the
                whole-state and subsampled g(r)
* ``export``    one XYZ frame and one snapshot world section
"""
from __future__ import annotations

import ctypes
import itertools
import math
from dataclasses import replace

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

from genesis_b200 import elements as E
from genesis_b200 import synth
from genesis_b200 import workloads as W
from genesis_b200._lib import Batch, Handle
from genesis_b200.adjoint import AdjointSpec, gr_loss, potential_loss
from genesis_b200.systems import GpuUniverse

SPACING = W.SPACING_FACTOR * max(E.SIGMA)
R_C = W.lattice_rc()
GRAVITY = 1e-3       # a constant whose pull is felt within a segment
LENS_JITTER = 0.12   # lattice disorder of a state handed to the lenses
GR_BINS = 256


# ------------------------------------------------------------------- cases


def listed() -> list[dict]:
    return [
        # the smallest universe that a scheduler drives tick by tick
        dict(name="host_tick_512", kind="host_tick", n=8, precision="mixed", coulomb=False, gravity=False,
             temperature=60.0, target=0.0),
        # the plain Lennard-Jones NVE run
        dict(name="nve_4096", kind="run", n=16, precision="mixed", coulomb=False, gravity=False, temperature=60.0,
             target=0.0, ticks=100, gr=False),
        # ionic NVT with the bond observation on every tick
        dict(name="ionic_observed_32768", kind="observed", n=32, precision="mixed", coulomb=True, gravity=False,
             temperature=300.0, target=300.0, ticks=10),
        # the reference's schedule of separate systems, charges and thermostat on
        dict(name="schedule_29791", kind="schedule", n=31, precision="mixed", coulomb=True, gravity=False,
             temperature=300.0, target=80.0, ticks=10),
        # every force term on, odd size
        dict(name="gravity_59319", kind="run", n=39, precision="mixed", coulomb=True, gravity=True,
             temperature=120.0, target=120.0, ticks=50, gr=True),
        # a drop-in system of a host-side world at an ordinary size
        dict(name="host_tick_262144", kind="host_tick", n=64, precision="mixed", coulomb=True, gravity=False,
             temperature=300.0, target=20.0),
        # the large condensation quench, sampled every 100 ticks
        dict(name="quench_2097152", kind="run", n=128, precision="mixed", coulomb=True, gravity=False,
             temperature=300.0, target=20.0, ticks=100, gr=True),
        # the plain FP64 path, odd size
        dict(name="fp64_250047", kind="run", n=63, precision="fp64", coulomb=True, gravity=False,
             temperature=300.0, target=20.0, ticks=10, gr=False),
        # the temperature sweep of 256 replicas
        dict(name="sweep_256", kind="sweep", replicas=256, lo=512, hi=16384, t_lo=20.0, t_hi=120.0, ticks=100),
        # sigma and epsilon gradients of both losses over a 200-tick horizon
        dict(name="adjoint_8000", kind="adjoint", n=20, precision="mixed", coulomb=False, temperature=60.0, ticks=200,
             every=20, initial=False),
        # structure analysis of one state
        dict(name="lens_262144", kind="lens", n=64, temperature=300.0),
        # one frame and one snapshot of the quench's state
        dict(name="export_250047", kind="export", n=63, temperature=300.0),
    ]


def _log(rng, lo: float, hi: float) -> float:
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _side(rng, lo: int, hi: int) -> int:
    """A lattice side whose atom count is spread over its logarithm."""
    return min(max(int(round(_log(rng, lo, hi))), lo), hi)


def draw(rng) -> dict:
    kind = rng.choice(["run", "run", "run", "host_tick", "host_tick", "observed", "schedule", "sweep", "adjoint",
                       "lens", "export"])
    t0 = round(rng.uniform(20.0, 300.0), 1)
    target = round(rng.uniform(20.0, 300.0), 1) if rng.random() < 0.6 else 0.0
    law = dict(coulomb=rng.random() < 0.6, gravity=rng.random() < 0.2)
    if kind == "run":
        precision = "fp64" if rng.random() < 0.3 else "mixed"
        n = _side(rng, 8, 80 if precision == "fp64" else 120)
        most = 10 if precision == "fp64" else 100
        return dict(kind=kind, n=n, precision=precision, **law, temperature=t0, target=target,
                    ticks=max(1, int(round(_log(rng, 1, most)))), gr=rng.random() < 0.4)
    if kind == "host_tick":
        return dict(kind=kind, n=_side(rng, 8, 100), precision="fp64" if rng.random() < 0.2 else "mixed", **law,
                    temperature=t0, target=target)
    if kind == "observed":
        return dict(kind=kind, n=_side(rng, 8, 64), precision="fp64" if rng.random() < 0.2 else "mixed", coulomb=True,
                    gravity=False, temperature=t0, target=target, ticks=rng.randint(1, 10))
    if kind == "schedule":
        return dict(kind=kind, n=_side(rng, 8, 64), precision="fp64" if rng.random() < 0.2 else "mixed", **law,
                    temperature=t0, target=target, ticks=rng.randint(1, 10))
    if kind == "sweep":
        hi = int(_log(rng, 1024, 16384))
        return dict(kind=kind, replicas=max(4, int(round(_log(rng, 4, 256)))), lo=512, hi=hi, t_lo=20.0,
                    t_hi=round(rng.uniform(40.0, 300.0), 1), ticks=rng.randint(10, 100))
    if kind == "adjoint":
        return dict(kind=kind, n=_side(rng, 8, 20), precision=rng.choice(["mixed", "fp64"]), coulomb=rng.random() < 0.4,
                    temperature=round(rng.uniform(20.0, 120.0), 1), ticks=rng.randint(20, 200),
                    every=rng.randint(5, 40), initial=rng.random() < 0.4)
    if kind == "lens":  # three cells of 3 r_c and more along each axis
        return dict(kind=kind, n=_side(rng, 19, 64), temperature=t0)
    return dict(kind=kind, n=_side(rng, 10, 80), temperature=t0)


# ------------------------------------------------------------- preparation


def _workload(case: dict, seed: int) -> W.Workload:
    observed = case["kind"] == "observed"
    target = case.get("target", 0.0)
    return W.Workload(case["kind"], n_side=case["n"], temperature=case["temperature"], steps=0, seed=seed,
                      electrostatics=case.get("coulomb", True), thermostat=target > 0.0,
                      thermostat_temperature=target if target > 0.0 else 300.0, bond_observation=observed,
                      bond_interaction=observed, species=(W.NA, W.O) if observed else None,
                      fixed_fractions={W.NA: 0.5, W.O: 0.5} if observed else None)


def _universe(case: dict, seed: int):
    """The configuration and the initial universe of a single-universe case."""
    wl = _workload(case, seed)
    cfg = wl.config()
    if case.get("gravity"):
        cfg.enable_gravity = True
        cfg.gravity_constant = GRAVITY
    if case["kind"] in ("lens", "export"):  # the disorder of a running state
        u = synth.lattice(case["n"], SPACING, LENS_JITTER, case["temperature"], cfg.thermal_constant, seed)
    else:
        u = wl.generate()
    return cfg, u


def _replicas(case: dict, seed: int) -> list[W.Workload]:
    """The sweep's sizes and temperatures go with the case, its universes with the seed."""
    reps = W.sweep_replicas(case["replicas"], 0, case["lo"], case["hi"], case["t_lo"], case["t_hi"])
    return [W.replica_workload(replace(r, seed=seed * 1000003 + k)) for k, r in enumerate(reps)]


def _pinned(n: int) -> np.ndarray:
    return torch.zeros((n, 3), dtype=torch.float64, pin_memory=True).numpy()


def _adjoint_spec(case: dict) -> AdjointSpec:
    return AdjointSpec(nsteps=case["ticks"], checkpoint_every=case["every"])


def _gr_target(spec: AdjointSpec) -> np.ndarray:
    """The pair distribution a fit aims at: a soft step at the contact distance."""
    r = (np.arange(spec.gr_bins) + 0.5) * spec.gr_rmax / spec.gr_bins
    return 1.0 / (1.0 + np.exp(-(r - 2.0) / 0.15))


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    if kind == "sweep":
        wls = _replicas(case, seed)
        b = Batch(wls[0].config(), [wl.config().size for wl in wls], [wl.thermostat_temperature for wl in wls])
        b.set_mode(4)  # the all-replica graph over neighbour lists
        b.set_universes([wl.generate() for wl in wls])
        n = int(b.natoms.sum())
        return dict(case=case, b=b, out=[_pinned(n) for _ in range(3)])
    cfg, u = _universe(case, seed)
    if kind == "schedule":
        return dict(case=case, u=GpuUniverse(cfg, u, case["precision"]))
    h = Handle(cfg, case.get("precision", "mixed"))
    h.set_universe(u)
    st = dict(case=case, h=h, cfg=cfg, out=[_pinned(u.n) for _ in range(3)], tick=0)
    if kind == "host_tick":
        st["out"][0][:], st["out"][1][:] = u.pos, u.vel
    if kind == "export":  # what the files are written from
        for name, each in (("frame", 64), ("world", 115)):
            st[name] = torch.zeros(64 + each * u.n, dtype=torch.uint8, pin_memory=True).numpy()
    if kind == "adjoint":
        st["spec"] = _adjoint_spec(case)
        st["target"] = _gr_target(st["spec"])
    return st


# --------------------------------------------------------------- one pass


def _columns(rec: np.ndarray) -> dict:
    return {f: np.ascontiguousarray(rec[f]) for f in rec.dtype.names}


def _state(st: dict) -> dict:
    st["h"].get_state_into(*st["out"])
    return dict(zip(("pos", "vel", "acc"), st["out"]))


def _address(a: np.ndarray):
    return a.ctypes.data_as(ctypes.POINTER(ctypes.c_double))


def run(st: dict):
    case = st["case"]
    kind = case["kind"]
    if kind == "sweep":
        b, (pos, vel, acc) = st["b"], st["out"]
        stats, _ = b.step(case["ticks"])
        b._check(b.lib.gx_batch_get_state(b.b, _address(pos), _address(vel), _address(acc)))
        return dict(stats=stats, pos=pos, vel=vel, acc=acc)
    if kind == "schedule":
        u = st["u"]
        u.run_ticks(case["ticks"])
        snap, w = u.resources["StatsSnapshot"], u.sync()
        return dict(kinetic=snap["kinetic"], potential=snap["energy_potential"], speed=snap["mean_speed"], pos=w.pos,
                    vel=w.vel, acc=w.acc)
    h = st["h"]
    if kind == "run":
        out = _columns(h.step(case["ticks"], stats=True, graph=True))
        if case["gr"]:
            counts, bins, _, _ = h.radial_distribution(3.0 * R_C, GR_BINS)
            out.update(counts=counts, bins=bins)
        return {**out, **_state(st)}
    if kind == "host_tick":
        rec = h.tick_host(*st["out"])
        return {**_columns(rec), **dict(zip(("pos", "vel", "acc"), st["out"]))}
    if kind == "observed":
        cfg = st["cfg"]
        for _ in range(case["ticks"]):
            h.step(1, stats=False, graph=True)
            st["tick"] += 1
            seen = h.bond_observe(cfg.bond_k_bind, cfg.bond_min_periods, st["tick"])
        return {**seen, **_state(st)}
    if kind == "adjoint":
        spec = st["spec"]
        V, g = h.adjoint_forward(spec.nsteps, **spec.kwargs())
        by_v = h.adjoint_backward(dl_dpotential=potential_loss(V)[1])
        by_g = h.adjoint_backward(dl_dgr=gr_loss(g, st["target"])[1], initial_state=case["initial"])
        return dict(potential=V, gr=g, by_potential=by_v, by_gr=by_g)
    if kind == "lens":
        labels, summary = h.clusters()
        counts, bins, _, _ = h.radial_distribution(3.0 * R_C, GR_BINS, 0)
        sample, sample_bins, _, _ = h.radial_distribution(3.0 * R_C, GR_BINS)
        return dict(labels=labels, summary=summary, counts=counts, bins=bins, sample=sample, sample_bins=sample_bins)
    frame, world, length = st["frame"], st["world"], [ctypes.c_size_t(), ctypes.c_size_t()]
    text = ctypes.cast(frame.ctypes.data, ctypes.c_char_p)
    h._check(h.lib.gx_xyz_frame(h.h, 0, text, len(frame), ctypes.byref(length[0])))
    h._check(h.lib.gx_snapshot_world(h.h, None, world.ctypes.data, len(world), ctypes.byref(length[1])))
    return dict(frame=frame, world=world, length=[x.value for x in length])


# -------------------------------------------------------------------- work


def _atoms(case: dict) -> float:
    if case["kind"] != "sweep":
        return float(case["n"]) ** 3
    lo, hi = float(case["lo"]), float(case["hi"])  # the mean of a log-uniform size
    return case["replicas"] * (hi - lo) / math.log(hi / lo) if hi > lo else case["replicas"] * lo


def work(case: dict) -> dict:
    """Bytes and operations of one pass: every tick reads and writes the three
    state columns (72 bytes an atom each way); a pair within the cutoff takes
    67 operations, 8 more with a second term, counted once."""
    n = _atoms(case)
    pairs = n * W.lattice_pairs_per_atom()
    kind = case["kind"]
    per_pair = 67.0 + (8.0 if case.get("coulomb") else 0.0) + (8.0 if case.get("gravity") else 0.0)
    if kind == "adjoint":  # forward, recomputation and two adjoint sweeps of about 200 operations a pair
        t = case["ticks"]
        return dict(bytes=t * n * 144.0, flops=t * pairs * (2 * per_pair + 2 * 200.0))
    if kind == "lens":  # every pair within each range: one distance (9) and one bin or union
        shell = 4.0 / 3.0 * math.pi / SPACING ** 3 / 2.0
        near = (E.BOND_FACTOR * max(E.SIGMA)) ** 3 * shell
        far = min((3.0 * R_C) ** 3, (0.5 * case["n"] * SPACING) ** 3) * shell
        return dict(bytes=n * (25.0 + 4.0), flops=n * (near + far) * 12.0)
    if kind == "export":  # positions, velocities, accelerations, mass, charge, element, id in; text and records out
        return dict(bytes=n * (93.0 + 35.0 + 115.0), flops=n * 50.0)
    t = case.get("ticks", 1)
    return dict(bytes=t * n * 144.0, flops=t * (pairs * per_pair + n * 30.0))


# ------------------------------------------------- the same in plain FP64


_HALF = [o for o in itertools.product((-1, 0, 1), repeat=3) if o > (0, 0, 0)]  # one of each pair of offsets


def _apart(d: torch.Tensor, L) -> torch.Tensor:
    return d - L * torch.round(d / L)


def _pairs_of_one(x: torch.Tensor, L: float, r: float, most: int = 1 << 25):
    """Chunks (i, j, distance) of every pair of one periodic universe within r, each once."""
    n, dev = len(x), x.device
    side = int(L // r)
    if n <= 5000 or side < 3:
        step = max(1, most // max(n, 1))
        for a in range(0, n, step):
            d = torch.linalg.vector_norm(_apart(x[a:a + step, None] - x[None], L), dim=-1)
            rows = torch.arange(a, min(a + step, n), device=dev)
            hit = (d < r) & (rows[:, None] < torch.arange(n, device=dev)[None])
            i, j = hit.nonzero(as_tuple=True)
            yield i + a, j, d[hit]
        return
    c = torch.clamp((torch.remainder(x + 0.5 * L, L) * (side / L)).long(), 0, side - 1)
    key = c[:, 0] + side * (c[:, 1] + side * c[:, 2])
    order = torch.argsort(key)
    count = torch.bincount(key, minlength=side ** 3)
    start = torch.cumsum(count, 0) - count
    widest = int(count.max())
    xs, cs = x[order], c[order]
    step = max(1, most // widest)
    for o in [(0, 0, 0)] + _HALF:
        for a in range(0, n, step):
            b = torch.remainder(cs[a:a + step] + torch.tensor(o, device=dev), side)
            B = b[:, 0] + side * (b[:, 1] + side * b[:, 2])
            q = start[B][:, None] + torch.arange(widest, device=dev)
            ok = q < (start[B] + count[B])[:, None]
            q = q.clamp(max=n - 1)
            p = torch.arange(a, min(a + step, n), device=dev)[:, None]
            if o == (0, 0, 0):
                ok &= q > p
            d = torch.linalg.vector_norm(_apart(xs[p] - xs[q], L), dim=-1)
            ok &= d < r
            i, k = ok.nonzero(as_tuple=True)
            yield order[i + a], order[q[i, k]], d[ok]


class _Reference:
    """The force schedule in plain FP64 for one or more universes side by side."""

    def __init__(self, cfg, universes, targets, device="cuda"):
        def put(of):
            return torch.from_numpy(np.concatenate([of(u) for u in universes])).to(device)

        self.cfg, self.targets = cfg, targets
        self.n = [u.n for u in universes]
        self.L = [float(u.box[0]) for u in universes]
        self.first = np.concatenate([[0], np.cumsum(self.n)])
        self.rep = torch.arange(len(self.n), device=device).repeat_interleave(torch.tensor(self.n, device=device))
        self.box = torch.tensor(self.L, dtype=torch.float64, device=device)[self.rep][:, None]
        self.x, self.v = put(lambda u: u.pos), put(lambda u: u.vel)
        self.a = torch.zeros_like(self.x)
        self.m, self.q, self.e = put(lambda u: u.mass), put(lambda u: u.charge), put(lambda u: u.elem).long()
        self.sigma = torch.tensor(cfg.sigma, dtype=torch.float64, device=device)
        self.eps = torch.tensor(cfg.epsilon_k, dtype=torch.float64, device=device)
        self.skin, self.moved, self.pairs = 1.0, math.inf, None

    def by_universe(self, per_atom: torch.Tensor) -> torch.Tensor:
        return torch.zeros(len(self.n), dtype=torch.float64, device=per_atom.device).index_add_(0, self.rep, per_atom)

    def cutoffs(self, sigma):
        top = sigma.max(0).values
        factors = E.LJ_CUTOFF_FACTOR, self.cfg.coulomb_cutoff, self.cfg.gravity_cutoff
        return [max(f, 1.0) * top for f in factors]

    def reach(self) -> float:
        lj, co, gr = (float(c) for c in self.cutoffs(self.sigma))
        return max(lj, co if self.cfg.enable_electrostatics else 0.0, gr if self.cfg.enable_gravity else 0.0)

    def list_pairs(self):
        """Pairs within the reach and a skin, renewed once atoms may have crossed half of it."""
        with torch.no_grad():
            self.moved += float(self.v.norm(dim=1).max()) * self.cfg.dt * 2.0
            if self.moved < self.skin:
                return
            self.moved, found = 0.0, []
            for k, L in enumerate(self.L):
                a, b = int(self.first[k]), int(self.first[k + 1])
                for i, j, _ in _pairs_of_one(self.x[a:b], L, self.reach() + self.skin):
                    found.append((i + a, j + a))
            self.pairs = (torch.cat([f[0] for f in found]), torch.cat([f[1] for f in found]))

    def forces(self, x, sigma, eps):
        """Accelerations, and per pair within reach its distance, energy and universe."""
        i, j = self.pairs
        dx = _apart(x[i] - x[j], self.box[i])
        d = torch.sqrt((dx * dx).sum(1))
        near = (d < self.reach()).nonzero()[:, 0]
        i, j, dx, d = i[near], j[near], dx[near], d[near]
        lj, co, gr = self.cutoffs(sigma)
        s = 0.5 * (sigma[self.e[i]] + sigma[self.e[j]])
        ep = self.cfg.thermal_constant * torch.sqrt(eps[self.e[i]] * eps[self.e[j]])
        r = torch.maximum(d, 0.5 * s)
        s6 = (s / r) ** 6
        v, f = 4.0 * ep * (s6 * s6 - s6), 24.0 * ep / s * (s / r) * (2.0 * s6 * s6 - s6)
        sw, dsw = self.switch(r, lj)
        inside = (d < lj).to(d)
        U, F = inside * v * sw, inside * (f * sw - v * dsw)
        terms = []
        if self.cfg.enable_electrostatics:
            terms.append((self.cfg.coulomb_constant * self.q[i] * self.q[j], co))
        if self.cfg.enable_gravity:
            terms.append((-self.cfg.gravity_constant * self.m[i] * self.m[j], gr))
        for strength, rc in terms:
            r = torch.clamp(d, min=0.5)
            v, f = strength / r, strength / (r * r)
            sw, dsw = self.switch(d, rc)
            inside = (d < rc).to(d)
            U, F = U + inside * v * sw, F + inside * (f * sw - v * dsw)
        push = dx * (F / d)[:, None]
        a = torch.zeros_like(x).index_add(0, i, push).index_add(0, j, -push) / self.m[:, None]
        return a, d, U, self.rep[i]

    @staticmethod
    def switch(r, rc):
        w = 0.1 * rc
        u = ((r - 0.9 * rc) / w).clamp(0.0, 1.0)
        return 1.0 - u ** 3 * (10.0 - 15.0 * u + 6.0 * u * u), -30.0 * u * u * (1.0 - u) ** 2 / w

    def move(self, x, v, a):
        dt = self.cfg.dt
        v = v + 0.5 * dt * a
        return torch.remainder(x + dt * v, self.box) - 0.5 * self.box, v

    def tick(self) -> dict:
        self.list_pairs()
        self.x, self.v = self.move(self.x, self.v, self.a)
        self.a, d, U, rep = self.forces(self.x, self.sigma, self.eps)
        self.v = self.v + 0.5 * self.cfg.dt * self.a
        K = self.by_universe(0.5 * self.m * (self.v * self.v).sum(1))
        lam = torch.ones_like(K)
        on = torch.tensor([t > 0.0 for t in self.targets], device=K.device)
        if self.cfg.enable_thermostat and bool(on.any()):
            n = torch.tensor(self.n, dtype=torch.float64, device=K.device)
            T = 2.0 / 3.0 * K / n / self.cfg.thermal_constant
            goal = torch.tensor(self.targets, dtype=torch.float64, device=K.device)
            scale = torch.sqrt(torch.clamp(1.0 + (goal / T - 1.0) / self.cfg.thermostat_tau, min=0.0))
            lam = torch.where(on, scale, lam)
            self.v = self.v * lam[self.rep][:, None]
        V = torch.zeros_like(K).index_add_(0, rep, U)
        return dict(kinetic=lam * lam * K, potential=V, pairs=torch.bincount(rep, minlength=len(self.n)),
                    speed_sum=self.by_universe(self.v.norm(dim=1)), **{"lambda": lam})


def _run_reference(ref: _Reference, ticks: int) -> dict:
    last = [ref.tick() for _ in range(ticks)]
    return {k: torch.stack([r[k] for r in last]) for k in last[0]}


def _exact_adjoint(case: dict, cfg, u):
    spec = _adjoint_spec(case)
    ref = _Reference(cfg, [u], [0.0])
    dev = ref.x.device
    sigma, eps = ref.sigma.clone().requires_grad_(), ref.eps.clone().requires_grad_()
    start = [t.clone().requires_grad_() for t in (ref.x, ref.v, ref.a)]
    centres = (torch.arange(spec.gr_bins, dtype=torch.float64, device=dev) + 0.5) * spec.gr_rmax / spec.gr_bins
    w = spec.gr_width
    shell = 4.0 * math.pi * centres ** 2 * math.sqrt(2.0 * math.pi) * w
    norm = float(np.prod(cfg.size)) / (0.5 * u.n * (u.n - 1) * shell)

    def one(x, v, a, s, e, i, j):
        ref.pairs = (i, j)
        x, v = ref.move(x, v, a)
        a, d, U, _ = ref.forces(x, s, e)
        d = d[d < spec.gr_rmax + spec.gr_support * w]
        z = d[:, None] - centres
        g = torch.where(z.abs() < spec.gr_support * w, torch.exp(-z * z / (2 * w * w)), 0.0).sum(0) * norm
        return x, v + 0.5 * cfg.dt * a, a, U.sum(), g

    x, v, a = start
    V, G = [], []
    for _ in range(spec.nsteps):
        ref.x, ref.v = x.detach(), v.detach()
        ref.moved += float(a.detach().norm(dim=1).max()) * cfg.dt * cfg.dt  # the kick that the list's test does not see
        ref.list_pairs()
        x, v, a, p, g = checkpoint(one, x, v, a, sigma, eps, *ref.pairs, use_reentrant=False)
        V.append(p)
        G.append(g)
    V, G = torch.stack(V), torch.stack(G).mean(0)
    by_v = torch.autograd.grad(V.mean(), [sigma, eps], retain_graph=True)
    loss = ((G - torch.from_numpy(_gr_target(spec)).to(dev)) ** 2).sum()
    by_g = torch.autograd.grad(loss, [sigma, eps] + start)
    by_g = [by_g[0], by_g[1], list(by_g[2:])] if case["initial"] else list(by_g[:2])
    return dict(potential=V.detach(), gr=G.detach(), by_potential=list(by_v), by_gr=by_g)


def _exact_gr(u, every: int) -> torch.Tensor:
    """g(r) over every `every`-th atom, whole strides only."""
    L, x = float(u.box[0]), torch.from_numpy(u.pos[::every][:u.n // every].copy()).cuda()
    r_max = min(3.0 * R_C, 0.5 * L)
    dr = r_max / GR_BINS
    counts = torch.zeros(GR_BINS, dtype=torch.float64, device="cuda")
    for _, _, d in _pairs_of_one(x, L, r_max):
        counts += torch.bincount((d / dr).long().clamp(max=GR_BINS - 1), minlength=GR_BINS)
    edge = torch.arange(GR_BINS + 1, dtype=torch.float64, device="cuda") * dr
    shell = 4.0 / 3.0 * math.pi * (edge[1:] ** 3 - edge[:-1] ** 3)
    return counts / (0.5 * len(x) * (len(x) - 1) * shell / L ** 3)


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind == "export":  # bytes
        return None
    if kind == "sweep":
        wls = _replicas(case, seed)
        ref = _Reference(wls[0].config(), [wl.generate() for wl in wls], [wl.thermostat_temperature for wl in wls])
        t = _run_reference(ref, case["ticks"])
        stats = torch.stack([t["kinetic"][-1], t["potential"][-1], t["lambda"][-1], t["pairs"][-1].double()], 1)
        return dict(stats=stats, pos=ref.x, vel=ref.v, acc=ref.a)
    cfg, u = _universe(case, seed)
    if kind == "lens":
        return dict(labels=None, summary=None, counts=None, bins=_exact_gr(u, 1), sample=None,
                    sample_bins=_exact_gr(u, u.n // E.G_SAMPLE_CAP + 1))
    if kind == "adjoint":
        return _exact_adjoint(case, cfg, u)
    ref = _Reference(cfg, [u], [case["target"]])
    t = _run_reference(ref, case.get("ticks", 1))
    state = dict(pos=ref.x, vel=ref.v, acc=ref.a)
    if kind == "observed":  # no bond lasts ten periods within a segment: the spring stays out of it
        return state
    if kind == "schedule":
        return dict(kinetic=float(t["kinetic"][-1, 0]), potential=float(t["potential"][-1, 0]),
                    speed=float(t["speed_sum"][-1, 0]) / u.n, **state)
    return {**{k: t[k][:, 0] for k in ("kinetic", "speed_sum", "potential", "lambda")}, **state}
