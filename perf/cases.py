"""The work that users of this framework have it do, as cases that can be timed and compared.

Four ways in, each through the public entry points of ``protomol3_b200``:

* ``md``: device-resident molecular dynamics, ``Integrator.run(n)``, then the state and the
  energies read back, as a program does at every output interval;
* ``host``: the drop-in call, ``SystemForce::evaluate`` / ``ForceGroup::evaluateSystemForces`` on
  host arrays, as a caller with its own integrator makes once per step;
* ``device``: ``pmb_evaluate_device`` on positions that are on the GPU already (one force term by
  itself, or a set);
* ``frames``: the same over several unrelated configurations in turn (re-evaluating the frames of
  a trajectory), so that every call builds its neighbour list anew.

The boxes are synthetic flexible TIP3P water at 1 g/cm^3 with Maxwell-Boltzmann velocities
(``protomol3_b200.waterbox``), of the sizes that the repository's tests, benchmark and serving
workload use.  Lengths are in A, energies in kcal/mol, timesteps in fs.
"""
import ctypes as C
import math

import numpy as np
import torch

from protomol3_b200 import _lib as L
from protomol3_b200 import constraints as CS
from protomol3_b200 import forces as F
from protomol3_b200 import waterbox as W

TIMEFACTOR = 48.88821290839616  # fs per internal time unit


def _case(**k):
    c = dict(mode="md", precision="mixed", waters=1000, boxes=1, waters_lo=0, terms="lj pme bonded", cutoff=9.0,
             switchon=7.5, order=4, gx=0, gy=0, gz=0, virial=False, steps=0, integrator="leapfrog", timestep=1.0,
             rigid=False, frames=0, pinned=False)
    unknown = set(k) - set(c) - {"name"}
    if unknown:
        raise ValueError("unknown keys %s" % sorted(unknown))
    c.update(k)
    if "pme" in c["terms"] and not c["gx"] and c["boxes"] == 1:
        c["gx"] = c["gy"] = c["gz"] = W.pme_grid_for(W.box_edge(c["waters"]))
    return c


def listed():
    return [
        # ProtoMol's own step on its smallest water fixture: one evaluate() on pageable host arrays
        # in the reference's FP64 arithmetic.  Latency and launches.
        _case(name="host_fp64_216", mode="host", precision="fp64", waters=216, cutoff=8.0, switchon=7.0),
        # a host integrator driving the 98,304-atom box, its arrays page-locked
        _case(name="host_mixed_98k", mode="host", waters=32768, cutoff=10.0, switchon=8.0, pinned=True),
        # a small NVE run with output every 25 steps: launch latency of the captured step
        _case(name="md_mixed_216", waters=216, cutoff=8.0, switchon=7.0, steps=25),
        # the 98,304-atom NVE run, output every 25 steps
        _case(name="md_mixed_98k", waters=32768, cutoff=10.0, switchon=8.0, steps=25),
        # an FP64 run of ordinary, ragged size
        _case(name="md_fp64_15k", precision="fp64", waters=5001, steps=25),
        # an ensemble of 256 uneven boxes (100 to 2,000 waters) advanced together; the smallest
        # need Ewald lattice images
        _case(name="md_mixed_ensemble_256", waters=2000, waters_lo=100, boxes=256, steps=10),
        # one Langevin segment of the serving workload (500 to 50,000 atoms), with the virial
        # for its pressure output
        _case(name="md_langevin_27k", waters=9001, integrator="langevin", virial=True, steps=25),
        # rigid water at 2 fs: SHAKE and RATTLE in every step
        _case(name="md_rigid_24k", waters=8000, rigid=True, timestep=2.0, steps=20),
        # energies, forces and virial of stored frames
        _case(name="frames_mixed_37k", mode="frames", waters=12345, frames=6, virial=True),
        # a PME force by itself, FP64, a higher order and an uneven grid
        _case(name="pme_fp64_order6_19k", mode="device", precision="fp64", waters=6400, terms="pme", order=6,
              gx=60, gy=64, gz=72, virial=True),
        # LennardJones and Coulomb by cutoff, C2 and C1 switched, without PME
        _case(name="cutoff_mixed_36k", mode="device", waters=12000, terms="lj coulomb", cutoff=10.0, switchon=8.0,
              virial=True),
        # the reciprocal sum alone, as a long-range force on its own (multiple time stepping)
        _case(name="recip_mixed_180k", mode="device", waters=60000, terms="recip", gx=125, gy=125, gz=125),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    mode = rng.choice(["md", "md", "md", "device", "device", "host", "frames"])
    rc = rng.choice([8.0, 9.0, 10.0, 12.0]) - rng.choice([0.0, 0.0, 0.25])
    c = dict(mode=mode, precision=rng.choice(["mixed", "mixed", "fp64"]), waters=_log_int(rng, 100, 33000),
             cutoff=rc, switchon=rc - rng.choice([0.5, 1.0, 1.5, 2.0]), order=rng.choice([4, 4, 4, 6, 8]),
             virial=rng.random() < 0.4)
    if mode == "md":
        if rng.random() < 0.35:  # several boxes in one system
            c["boxes"] = _log_int(rng, 2, 128)
            c["waters_lo"] = _log_int(rng, 100, 300)
            c["waters"] = c["waters_lo"] + _log_int(rng, 10, 1500)
            c["precision"] = "mixed"
        atoms = 3 * c["waters"] * c.get("boxes", 1)
        c["steps"] = rng.randint(5, max(6, min(25, 1500000 // atoms)))
        c["integrator"] = rng.choice(["leapfrog", "leapfrog", "langevin"])
        c["rigid"] = c.get("boxes", 1) == 1 and rng.random() < 0.25
        c["timestep"] = 2.0 if c["rigid"] else rng.choice([0.5, 1.0])
    elif mode == "host":
        c["pinned"] = rng.random() < 0.5
    elif mode == "device":
        c["terms"] = rng.choice(["lj pme bonded", "lj", "lj coulomb", "pme", "recip", "pme bonded"])
    else:
        c["frames"] = rng.randint(2, 6)
    if c.get("boxes", 1) == 1 and rng.random() < 0.5:  # an uneven grid, finer or coarser than 1 A
        edge = W.box_edge(c["waters"])
        for k in ("gx", "gy", "gz"):
            c[k] = min(135, W.pme_grid_for(edge, rng.uniform(0.75, 1.25)))
    return _case(**c)


# ------------------------------------------------------------------------------------ inputs
def _box(case, waters, seed):
    """A water box; the bonds and angles of flexible water vibrate (0.02 A per axis is what 300 K
    gives), rigid water starts at its rest geometry."""
    b = W.water_box(waters, seed=seed)
    if not case["rigid"]:
        b["pos"] = b["pos"] + np.random.default_rng([seed, 1]).normal(0.0, 0.02, b["pos"].shape)
    return b


def _boxes(case, seed):
    """The boxes of a case, made from the seed alone."""
    n, lo = case["waters"], case["waters_lo"]
    if case["boxes"] == 1:
        return [_box(case, n, seed)]
    counts = np.random.default_rng(4321).integers(lo, n + 1, size=case["boxes"])  # the case's sizes, whatever the seed
    return [_box(case, int(w), seed * 1000 + 1 + k) for k, w in enumerate(counts)]


def _grids(case, boxes):
    if case["gx"]:
        return [(case["gx"], case["gy"], case["gz"])]
    return [(W.pme_grid_for(b["box"][0]),) * 3 for b in boxes]


def _frames(case, boxes, seed):
    """Positions of every configuration: the box's, or that many boxes of the same size."""
    if case["mode"] != "frames":
        return [np.concatenate([b["pos"] for b in boxes])]
    return [_box(case, case["waters"], seed + 7919 * k)["pos"] for k in range(case["frames"])]


def _force_list(case, grids):
    terms, rc = case["terms"].split(), case["cutoff"]
    fl = []
    lj = ("C2", case["switchon"], rc) if "lj" in terms else None
    if lj or "coulomb" in terms:
        fl.append(F.NonbondedCutoffSystemForce(lj=lj, coulomb=("C1", 0.0, rc) if "coulomb" in terms else None))
    if "pme" in terms or "recip" in terms:
        whole = "pme" in terms
        one = len(grids) == 1
        fl.append(F.NonbondedPMEwaldSystemForce(grids[0] if one else (0, 0, 0), rc, order=case["order"], real=whole,
                                                correction=whole, box_grids=None if one else grids))
    if "bonded" in terms:
        fl.append(F.BondedSystemForce())
    return fl


_STREAM = []


def _stream():
    """The program's own stream (one for all of its device evaluations)."""
    if not _STREAM:
        _STREAM.append(torch.cuda.Stream())
    return _STREAM[0]


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.mode, s.virial, s.steps = case["mode"], case["virial"], case["steps"]
    boxes = _boxes(case, seed)
    s.topo = F.Topology(boxes, case["precision"])
    s.forces = _force_list(case, _grids(case, boxes))
    frames = _frames(case, boxes, seed)
    n = s.topo.n_atoms
    if s.mode == "md":
        s.md = F.Integrator(s.topo, s.forces, timestep=case["timestep"], kind=case["integrator"], temperature=300.0,
                            gamma=1.0, seed=seed)
        if case["virial"]:
            s.md.set_virial(True)
        if case["rigid"]:
            s.md.set_constraints(CS.rattle_shake_constraints(boxes[0]))
        s.md.set_state(frames[0], np.concatenate([b["vel"] for b in boxes]))
    elif s.mode == "host":
        if case["pinned"]:
            s.keep = [torch.empty((n, 3), dtype=torch.float64, pin_memory=True) for _ in range(2)]
            s.pos, s.frc = (t.numpy() for t in s.keep)
        else:
            s.pos, s.frc = np.empty((n, 3)), np.empty((n, 3))
        s.pos[:] = frames[0]
        s.energies = F.ScalarStructure(len(boxes), virial=s.virial)
    else:
        stream = _stream()
        s.topo.set_stream(stream.cuda_stream)
        with torch.cuda.stream(stream):
            s.pos = torch.from_numpy(np.stack(frames)).cuda()
            s.frc = torch.zeros_like(s.pos)
            s.energies = torch.zeros((len(frames), len(boxes), L.E_STRIDE), dtype=torch.float64, device="cuda")
        stream.synchronize()
        s.handles = (C.c_void_p * len(s.forces))(*[f.handle(s.topo) for f in s.forces])
    return s


def run(s):
    if s.mode == "md":
        s.md.run(s.steps)
        pos, vel = s.md.state()
        energies, kinetic = s.md.energies()
        return {"positions": pos, "velocities": vel, "energies": energies, "kinetic": kinetic}
    if s.mode == "host":
        s.frc[:] = 0.0
        s.energies.clear()
        F.evaluate_all(s.topo, s.forces, s.pos, s.frc, s.energies)
        return {"forces": s.frc, "energies": s.energies.table}
    system, lib = s.topo.system(), L.lib()
    for k in range(s.pos.shape[0]):
        L.check(lib.pmb_evaluate_device(system, C.addressof(s.handles), len(s.forces), s.pos[k].data_ptr(),
                                        s.frc[k].data_ptr(), s.energies[k].data_ptr(), int(s.virial)))
    return {"forces": s.frc, "energies": s.energies}


# ------------------------------------------------------------------------- what a pass needs
def work(case):
    """Positions, velocities and topology in, forces or the new state out, once per pass; pairs
    within the cutoff at 70 operations, the transforms at 5 n log2 n, the stencils at 8 a point."""
    evaluations = max(1, case["steps"], case["frames"])
    terms = case["terms"].split()
    sizes = [case["waters"]] if case["boxes"] == 1 else \
        np.linspace(case["waters_lo"], case["waters"], case["boxes"]).astype(int).tolist()
    flops = 0.0
    for k, w in enumerate(sizes):
        n, edge = 3.0 * w, W.box_edge(w)
        if "lj" in terms or "coulomb" in terms or "pme" in terms:
            flops += 70.0 * 0.5 * n * min(n, 4.0 / 3.0 * math.pi * case["cutoff"] ** 3 * n / edge ** 3)
        if "pme" in terms or "recip" in terms:
            g = (case["gx"], case["gy"], case["gz"]) if case["gx"] else (W.pme_grid_for(edge),) * 3
            points = float(g[0] * g[1] * g[2])
            flops += 5.0 * points * math.log2(points) + 16.0 * n * case["order"] ** 3
        if "bonded" in terms:
            flops += 60.0 * n
    atoms = 3.0 * sum(sizes)
    if case["mode"] == "md":
        moved = atoms * (24 * 4 + 8 + 8 + 4 + 4)  # positions and velocities in and out; mass, charge, type, molecule
    else:
        moved = atoms * max(1, case["frames"]) * (24 + 24) + atoms * (8 + 4 + 4)
    return {"bytes": moved, "flops": flops * evaluations}


def tolerance(case):
    """About four times and more of what another order of the sums shows (other sort cells and
    another list radius, two passes): FP64 forces differ by 2e-13 and energies, rounded to 2^-32
    kcal/mol and small differences of large terms, by up to 5e-11; mixed forces by 1.1e-6 of their
    norm (2.6e-5 of the RMS force at one atom), the velocities of a run by 9e-7 (1.3e-5), of a rigid
    run by 5e-6 (2.3e-4)."""
    if case["precision"] == "fp64":
        return {"rel": 1e-9, "max": 1e-8}
    if case["mode"] == "md" and case["rigid"]:
        return {"rel": 2e-5, "max": 1e-3}
    return {"rel": 1e-5, "max": 2e-4}


# ------------------------------------------------------------------------------ in 64 bits
def _alpha(rc, accuracy=1e-6):
    hi = 1.0
    while math.erfc(hi * rc) / rc >= accuracy:
        hi *= 2.0
    lo = 0.0
    for _ in range(100):
        a = 0.5 * (lo + hi)
        if math.erfc(a * rc) / rc >= accuracy:
            lo = a
        else:
            hi = a
    return a


def _erfc_poly(x):
    """Abramowitz & Stegun 7.1.26 without its exponential: what the real-space term is defined by."""
    t = 1.0 / (1.0 + 0.3275911 * x)
    return t * (0.254829592 + t * (-0.284496736 + t * (1.421413741 + t * (-1.453152027 + t * 1.061405429))))


def _spline(order, w):
    """Cardinal B-spline weights and derivatives at the fractions w: [order, n] each."""
    th = [1.0 - w, w]
    for k in range(2, order):
        if k == order - 1:
            low = list(th)
        div, prev = 1.0 / k, th
        th = [div * (1.0 - w) * prev[0]]
        for j in range(1, k):
            th.append(div * ((w + (k - j)) * prev[j - 1] + (j + 1 - w) * prev[j]))
        th.append(div * w * prev[k - 1])
    if order == 2:
        return torch.stack(th), torch.stack([-torch.ones_like(w), torch.ones_like(w)])
    zero = torch.zeros_like(w)
    low = [zero] + low + [zero]
    return torch.stack(th), torch.stack([low[j] - low[j + 1] for j in range(order)])


class _Exact:
    """Forces of one box in FP64, from the definitions."""

    def __init__(self, case, box, grid):
        self.case, self.grid = case, grid
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        t = lambda a, d=torch.float64: torch.from_numpy(np.ascontiguousarray(a)).to(self.dev, d)  # noqa: E731
        self.L, self.q, self.n = t(box["box"]), t(box["charge"]), len(box["charge"])
        self.type, self.mol = t(box["type"], torch.int64), t(box["molecule"], torch.int64)
        self.lj = t(box["lj"])
        self.excl = t(box["excl_pairs"], torch.int64)
        self.bonds, self.bk, self.br = t(box["bonds"], torch.int64), t(box["bond_k"]), t(box["bond_r0"])
        self.angles, self.ak, self.at = t(box["angles"], torch.int64), t(box["angle_k"]), t(box["angle_theta0"])
        self.mass = t(box["mass"])[:, None]
        self.terms = case["terms"].split()
        self.alpha = _alpha(case["cutoff"])
        self.pairs = self.pairs_at = None
        rc, e = case["cutoff"], [float(v) for v in box["box"]]
        reach = [int(math.floor(rc / v + 1.0)) for v in e]
        lat = [(a * e[0], b * e[1], c * e[2]) for a in range(-reach[0], reach[0] + 1)
               for b in range(-reach[1], reach[1] + 1) for c in range(-reach[2], reach[2] + 1) if a or b or c]
        self.images = [v for v in lat if math.sqrt(v[0] ** 2 + v[1] ** 2 + v[2] ** 2) <= 2 * rc]
        if grid is not None:
            self._tables()

    def _wrap(self, d):
        return d - self.L * torch.round(d / self.L)

    def _find_pairs(self, pos, margin):
        """Pairs i < j within the cutoff and a margin, excluded ones left out (all of them where
        the box is too small for the nearest image alone)."""
        n, r2max = self.n, (self.case["cutoff"] + margin) ** 2
        got, step = [], max(1, 200_000_000 // n)
        index = torch.arange(n, device=self.dev)
        for i0 in range(0, n, step):
            i = index[i0:i0 + step]
            r2 = torch.zeros((len(i), n), dtype=torch.float64, device=self.dev)
            for k in range(3):
                d = pos[None, :, k] - pos[i, None, k]
                d -= self.L[k] * torch.round(d / self.L[k])
                r2 += d * d
            near = (r2 <= r2max) if not self.images else torch.ones_like(r2, dtype=torch.bool)
            a, b = torch.nonzero(near & (index[None, :] > i[:, None]), as_tuple=True)
            got.append(torch.stack([a + i0, b]))
        pairs = torch.cat(got, 1)
        return pairs, self.mol[pairs[0]] == self.mol[pairs[1]]

    def _pair_terms(self, pos, f, e, vir):
        if not ({"lj", "coulomb", "pme"} & set(self.terms)):
            return
        moved = math.inf if self.pairs is None else float((pos - self.pairs_at).abs().max())
        if moved > 0.4:
            self.pairs, self.same = self._find_pairs(pos, 1.5 if self.case["steps"] else 0.0)
            self.pairs_at = pos.clone()
        c, (i, j) = self.case, self.pairs
        base = self._wrap(pos[j] - pos[i])
        rc2 = c["cutoff"] ** 2
        qq = self.q[i] * self.q[j]
        for image in [None] + (self.images if "pme" in self.terms else []):
            d = base if image is None else base + torch.tensor(image, dtype=torch.float64, device=self.dev)
            r2 = (d * d).sum(1)
            keep = r2 <= rc2
            if image is None:
                keep &= ~self.same
            d, r2, ii, jj, q = d[keep], r2[keep], i[keep], j[keep], qq[keep]
            r = torch.sqrt(r2)
            fs = torch.zeros_like(r2)
            if "lj" in self.terms and image is None:
                ab = self.lj[self.type[ii], self.type[jj]]
                r6 = 1.0 / r2 ** 3
                en = ab[:, 0] * r6 * r6 - ab[:, 1] * r6
                fo = (12.0 * ab[:, 0] * r6 * r6 - 6.0 * ab[:, 1] * r6) / r2
                ron2 = c["switchon"] ** 2
                w = (rc2 - ron2) ** 3
                c2 = rc2 - r2
                c4 = c2 * (rc2 - 3.0 * ron2 + 2.0 * r2)
                on = r2 >= ron2
                val = torch.where(on, c2 * c4 / w, torch.ones_like(r2))
                der = torch.where(on, 4.0 / w * (c2 * c2 - c4), torch.zeros_like(r2))
                fs = fs + fo * val - en * der
                e[1] += (en * val).sum()
            if "coulomb" in self.terms:
                rc = c["cutoff"]
                en = q / r
                val = 1.0 - r * (1.5 / rc - r2 * 0.5 / rc ** 3)
                der = -1.5 / rc / r + r * 1.5 / rc ** 3
                fs = fs + en / r2 * val - en * der
                e[0] += (en * val).sum()
            if "pme" in self.terms:
                g = q * torch.exp(-self.alpha ** 2 * r2)
                en = _erfc_poly(self.alpha * r) * g / r
                fs = fs + (en + 2.0 * self.alpha / math.sqrt(math.pi) * g) / r2
                e[0] += en.sum()
            fv = d * fs[:, None]
            f.index_add_(0, jj, fv)
            f.index_add_(0, ii, -fv)
            vir += fv.T @ d

    def _tables(self):
        order, bs, ms = self.case["order"], [], []
        at0 = _spline(order, torch.zeros(1, dtype=torch.float64, device=self.dev))[0][:, 0]
        for k, n in enumerate(self.grid):
            i = torch.arange(n, dtype=torch.float64, device=self.dev)
            x = 2.0 * math.pi * i[:, None] * torch.arange(order, device=self.dev)[None, :] / n
            b = 1.0 / ((at0 * torch.cos(x)).sum(1) ** 2 + (at0 * torch.sin(x)).sum(1) ** 2)
            m = torch.where(i <= n // 2, i, i - n) / self.L[k]
            bs.append(b)
            ms.append(m)
        m2 = ms[0][:, None, None] ** 2 + ms[1][None, :, None] ** 2 + ms[2][None, None, :] ** 2
        m2[0, 0, 0] = 1.0
        th = bs[0][:, None, None] * bs[1][None, :, None] * bs[2][None, None, :] * \
            torch.exp(-(math.pi / self.alpha) ** 2 * m2) / (math.pi * self.L.prod() * m2)
        th[0, 0, 0] = 0.0
        self.ms, self.m2, self.theta = ms, m2, th

    def _reciprocal(self, pos, f, e, vir):
        order, g = self.case["order"], self.grid
        th, dth, at = [], [], []
        for k in range(3):
            u = pos[:, k] / self.L[k]
            u = (u - torch.floor(u)) * g[k]
            cell = torch.floor(u)
            a, b = _spline(order, u - cell)
            th.append(a)
            dth.append(b * (g[k] / self.L[k]))
            at.append((cell.long()[None, :] + torch.arange(order, device=self.dev)[:, None] - (order - 1) // 2) % g[k])
        grid = torch.zeros(g[0] * g[1] * g[2], dtype=torch.float64, device=self.dev)
        where = [[(at[0][a] * g[1] + at[1][b])[None, :] * g[2] + at[2] for b in range(order)] for a in range(order)]
        for a in range(order):
            for b in range(order):
                grid.index_add_(0, where[a][b].reshape(-1), (self.q * th[0][a] * th[1][b] * th[2]).reshape(-1))
        spec = torch.fft.fftn(grid.reshape(g))
        en = 0.5 * self.theta * (spec.real ** 2 + spec.imag ** 2)
        e[0] += en.sum()
        v = 2.0 * (1.0 / self.m2 + (math.pi / self.alpha) ** 2)
        m = [self.ms[0][:, None, None], self.ms[1][None, :, None], self.ms[2][None, None, :]]
        for a in range(3):
            vir[a, a] += en.sum()
            for b in range(3):
                vir[a, b] -= (en * v * m[a] * m[b]).sum()
        phi = (torch.fft.ifftn(spec * self.theta).real * grid.numel()).reshape(-1)
        for a in range(order):
            for b in range(order):
                p = phi[where[a][b]]
                s, ds = (p * th[2]).sum(0) * self.q, (p * dth[2]).sum(0) * self.q
                f[:, 0] -= dth[0][a] * th[1][b] * s
                f[:, 1] -= th[0][a] * dth[1][b] * s
                f[:, 2] -= th[0][a] * th[1][b] * ds

    def _correction(self, pos, f, e, vir):
        i, j = self.excl[:, 0], self.excl[:, 1]
        d = self._wrap(pos[j] - pos[i])
        r2 = (d * d).sum(1)
        r, qq = torch.sqrt(r2), self.q[i] * self.q[j]
        en = torch.erf(self.alpha * r) / r
        e[0] -= (qq * en).sum()
        fs = qq * (2.0 * self.alpha / math.sqrt(math.pi) * torch.exp(-self.alpha ** 2 * r2) - en) / r2
        fv = d * fs[:, None]
        f.index_add_(0, j, fv)
        f.index_add_(0, i, -fv)
        vir += fv.T @ d

    def _bonded(self, pos, f, e, vir):
        a, b = self.bonds[:, 0], self.bonds[:, 1]
        d = self._wrap(pos[a] - pos[b])
        r = d.norm(dim=1)
        x = r - self.br
        fv = d * (-2.0 * self.bk * x / r)[:, None]
        f.index_add_(0, a, fv)
        f.index_add_(0, b, -fv)
        e[2] += (self.bk * x * x).sum()
        vir += fv.T @ d
        a, b, c = self.angles[:, 0], self.angles[:, 1], self.angles[:, 2]
        u, w = self._wrap(pos[a] - pos[b]), self._wrap(pos[c] - pos[b])
        lu, lw = u.norm(dim=1, keepdim=True), w.norm(dim=1, keepdim=True)
        theta = torch.atan2(torch.linalg.cross(u, w).norm(dim=1), (u * w).sum(1))
        x = theta - self.at
        k = (2.0 * self.ak * x / torch.sin(theta))[:, None]
        cos = torch.cos(theta)[:, None]
        fa = -k * (u / lu * cos - w / lw) / lu
        fc = -k * (w / lw * cos - u / lu) / lw
        f.index_add_(0, a, fa)
        f.index_add_(0, c, fc)
        f.index_add_(0, b, -fa - fc)
        e[3] += (self.ak * x * x).sum()
        vir += fa.T @ u + fc.T @ w

    def constants(self):
        """Self energy and a charge's own images: what the host call and the MD energies add."""
        e, vir = 0.0, np.zeros((3, 3))
        if "pme" not in self.terms:
            return e, vir
        q2, a = float((self.q ** 2).sum()), self.alpha
        e -= q2 * a / math.sqrt(math.pi)
        for v in self.images:
            r2 = v[0] ** 2 + v[1] ** 2 + v[2] ** 2
            if r2 > self.case["cutoff"] ** 2:
                continue
            r = math.sqrt(r2)
            g = math.exp(-a * a * r2)
            en = _erfc_poly(a * r) * g / r
            e += q2 * en
            vir += q2 * (en + 2.0 * a / math.sqrt(math.pi) * g) / r2 * np.outer(v, v)
        return e, vir

    def forces(self, pos):
        """Forces and the row [Coulomb, LJ, bond, angle, virial (9), 0, 0, 0] of energies."""
        f = torch.zeros_like(pos)
        e = torch.zeros(4, dtype=torch.float64, device=self.dev)
        vir = torch.zeros((3, 3), dtype=torch.float64, device=self.dev)
        self._pair_terms(pos, f, e, vir)
        if "pme" in self.terms or "recip" in self.terms:
            self._reciprocal(pos, f, e, vir)
        if "pme" in self.terms:
            self._correction(pos, f, e, vir)
        if "bonded" in self.terms:
            self._bonded(pos, f, e, vir)
        row = np.zeros(16)
        row[:4] = e.cpu().numpy()
        if self.case["virial"]:
            row[4:13] = vir.reshape(-1).cpu().numpy()
        return f, row

    def with_constants(self, row):
        e, vir = self.constants()
        row[0] += e
        if self.case["virial"]:
            row[4:13] += vir.reshape(-1)
        return row


def exact(case, seed):
    if case["mode"] == "md" and (case["rigid"] or case["integrator"] != "leapfrog"):
        return None  # the constraint sweeps' stopping rule, and the noise, are the framework's own
    boxes = _boxes(case, seed)
    grids = _grids(case, boxes) if "pme" in case["terms"] or "recip" in case["terms"] else [None] * len(boxes)
    systems = [_Exact(case, b, grids[k]) for k, b in enumerate(boxes)]
    on = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(systems[0].dev)  # noqa: E731
    if case["mode"] != "md":
        out_f, out_e = [], []
        for frame in _frames(case, boxes, seed):
            systems[0].pairs = None
            f, row = systems[0].forces(on(frame))
            out_f.append(f.cpu().numpy())
            out_e.append((systems[0].with_constants(row) if case["mode"] == "host" else row)[None])
        if case["mode"] == "host":
            return {"forces": out_f[0], "energies": out_e[0]}
        return {"forces": np.stack(out_f), "energies": np.stack(out_e)}
    h = case["timestep"] / TIMEFACTOR
    out = {"positions": [], "velocities": [], "energies": [], "kinetic": []}
    for s, b in zip(systems, boxes):
        x, v = on(b["pos"]).clone(), on(b["vel"]).clone()
        f, _ = s.forces(x)
        v += f * (0.5 * h) / s.mass
        for k in range(case["steps"]):
            x += v * h
            f, row = s.forces(x)
            v += f * (h if k + 1 < case["steps"] else 0.5 * h) / s.mass
        out["positions"].append(x.cpu().numpy())
        out["velocities"].append(v.cpu().numpy())
        out["energies"].append(s.with_constants(row)[None])
        out["kinetic"].append([float(0.5 * (s.mass * v * v).sum())])
        s.pairs = s.pairs_at = s.same = None
    return {k: np.concatenate([np.asarray(a) for a in v]) for k, v in out.items()}
