"""The workloads whose speed is measured, each through the public Python entry points.

A user of this package does one of three things: replaces a host MD code's
force call (``forces_midpoint_all`` once, or ``MidpointLJ.forces_at`` every
step with the caller's own host arrays), runs velocity-Verlet steps on the
device (``MidpointLJ.run``), or runs a batch of independent boxes.  The listed
cases are these three at the sizes of the package's configurations (the
32,000-atom crystal, the 1,048,576-atom liquid, the slab in vapour, the
512-box ensemble, the 16,777,216-atom binary mixture) and at smaller and odd
ones; ``draw`` gives others of the same ranges.

A pass of mode "call" is one ``forces_at`` at new positions of atoms that the
context has held since its start; "oneshot" is one ``forces_midpoint_all``
(context made and freed inside); "run" loads a configuration into the context
that the program keeps (``set_atoms``), runs its steps and reads the result.

A case is a dict of plain values:
  mode       "call", "oneshot" or "run"
  lattice    "fcc" (4 m^3 atoms), "sc" (m^3), "mix" (sc, two types 80:20),
             "slab" (m^3 liquid sites and vapour around them), "ensemble"
  m, boxes   sites per edge; boxes of an ensemble
  rho, temp, jitter (of the lattice spacing), rc, potential
  precision, skin (0: no pair lists), tile (0: the library's), balance
  steps, dt  of a run; energy: energies are asked for; accumulate: += call
  pinned     the caller's arrays are page-locked (those of a run always are)
  out        what a run returns: "state" (positions, velocities) or "forces"
"""
import math

import numpy as np
import torch

import examd_gb300 as ex

# Kob-Andersen-type table of the binary mixture (eps, sigma; cutoff rc sigma per pair)
MIX_EPS = ((1.0, 1.5), (1.5, 0.5))
MIX_SIGMA = ((1.0, 0.8), (0.8, 0.88))
CHUNK = 20  # steps per CUDA graph of a run, as the package's examples use

BASE = {"mode": "call", "lattice": "fcc", "m": 20, "boxes": 1, "rho": 0.8442, "temp": 1.0, "jitter": 0.09, "rc": 2.5,
        "potential": "lj", "precision": "fp64", "skin": 0.0, "tile": 0, "balance": 0, "steps": 0, "dt": 0.005,
        "energy": False, "accumulate": False, "pinned": False, "out": "forces"}


def _case(**kw):
    return dict(BASE, **kw)


def listed():
    return [
        # the smallest call: a driver's force call for 1,000 atoms of a gas, the reference's += into its own array
        _case(name="gas1k_fp64_call", lattice="sc", m=10, rho=0.5, jitter=0.2, energy=True, accumulate=True),
        # the drop-in routine called once, as the reference's driver does (context made and freed inside)
        _case(name="fcc9k_fp64_oneshot", mode="oneshot", m=13, energy=True),
        # the 32,000-atom FCC crystal, NVE steps with energies every step, in both precision forms
        _case(name="fcc32k_fp64_run", mode="run", m=20, temp=0.72, jitter=0.0, steps=101, energy=True, out="state"),
        _case(name="fcc32k_mixed_run", mode="run", m=20, temp=0.72, jitter=0.0, steps=101, energy=True, out="state",
              precision="mixed"),
        # FP64 force call of an odd-sized binary mixture in ordinary (pageable) numpy arrays
        _case(name="mix104k_fp64_call", lattice="mix", m=47, rho=1.2, jitter=0.1, energy=True),
        # FP64 force call of the 1,048,576-atom liquid with the driver's page-locked arrays
        _case(name="liquid1m_fp64_call", m=64, pinned=True),
        # mixed-form force call without pair lists, long cutoff, odd size, energy and virial
        _case(name="liquid276k_rc3_mixed_call", m=41, rc=3.0, precision="mixed", energy=True, pinned=True),
        # steps of the 1,048,576-atom liquid on pair lists at the tiles the autotuner picks for it
        _case(name="liquid1m_lists_run", mode="run", m=64, precision="mixed", skin=0.4, tile=6, balance=1, steps=61),
        # uneven density: a liquid slab in vapour in an elongated box, long cutoff, pair lists, default tiles
        _case(name="slab533k_lists_run", mode="run", lattice="slab", m=79, rho=0.75, temp=0.85, jitter=0.12, rc=3.0,
              precision="mixed", skin=0.5, steps=61),
        # a batch of 512 boxes of 256 to 16,384 atoms, energies of every box at every step
        _case(name="ensemble512_mixed_run", mode="run", lattice="ensemble", boxes=512, precision="mixed", steps=41,
              energy=True),
        # the driver's force call on pair lists between two rebuilds, 2,097,152 atoms, page-locked arrays
        _case(name="mix2m_lists_call", lattice="mix", m=128, rho=1.2, jitter=0.1, precision="mixed", skin=0.4,
              pinned=True),
        # the largest configuration: steps of the 16,777,216-atom mixture on pair lists
        _case(name="mix17m_lists_run", mode="run", lattice="mix", m=256, rho=1.2, jitter=0.1, precision="mixed",
              skin=0.4, tile=5, steps=21, dt=0.003),
    ]


def _between(rng, lo, hi):
    """A whole number in [lo, hi], spread over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("gas", "oneshot", "run64", "run32", "mix64", "liquid64", "liquid32", "lists", "slab",
                       "ensemble", "mixcall", "mixrun"))
    if kind == "gas":
        return _case(lattice="sc", m=_between(rng, 9, 16), rho=round(rng.uniform(0.3, 0.7), 3), jitter=0.2, energy=True,
                     accumulate=rng.random() < 0.5, precision=rng.choice(("fp64", "mixed")))
    if kind == "oneshot":
        return _case(mode="oneshot", m=_between(rng, 8, 25), rho=round(rng.uniform(0.6, 0.9), 3), energy=True,
                     precision=rng.choice(("fp64", "mixed")))
    if kind in ("run64", "run32"):
        return _case(mode="run", m=_between(rng, 10, 40), temp=round(rng.uniform(0.5, 1.2), 3), jitter=0.0,
                     steps=rng.choice((61, 81, 101)), energy=rng.random() < 0.5, out="state",
                     precision="fp64" if kind == "run64" else "mixed")
    if kind == "mix64":
        return _case(lattice="mix", m=_between(rng, 20, 100), rho=1.2, jitter=0.1, energy=rng.random() < 0.5,
                     pinned=rng.random() < 0.5)
    if kind == "liquid64":
        return _case(m=_between(rng, 16, 64), rho=round(rng.uniform(0.6, 0.9), 3), pinned=True,
                     rc=rng.choice((2.5, 3.0)), energy=rng.random() < 0.3)
    if kind == "liquid32":
        return _case(m=_between(rng, 16, 80), rho=round(rng.uniform(0.6, 0.9), 3), pinned=rng.random() < 0.7,
                     rc=rng.choice((2.5, 3.0)), precision="mixed", energy=rng.random() < 0.5,
                     potential=rng.choice(("lj", "lj", "lj_shifted", "wca")))
    if kind == "lists":
        return _case(mode="run", m=_between(rng, 24, 96), rho=round(rng.uniform(0.6, 0.9), 3), precision="mixed",
                     skin=rng.choice((0.3, 0.4, 0.5)), tile=rng.choice((0, 5, 6)), balance=rng.randint(0, 1),
                     rc=rng.choice((2.5, 3.0)), steps=rng.choice((41, 61)), energy=rng.random() < 0.3)
    if kind == "slab":
        return _case(mode="run", lattice="slab", m=_between(rng, 40, 100), rho=0.75, temp=0.85, jitter=0.12, rc=3.0,
                     precision="mixed", skin=rng.choice((0.0, 0.4, 0.5)), steps=61)
    if kind == "ensemble":
        return _case(mode="run", lattice="ensemble", boxes=_between(rng, 16, 512),
                     precision=rng.choice(("mixed", "mixed", "fp64")), steps=41, energy=rng.random() < 0.7)
    if kind == "mixcall":
        return _case(lattice="mix", m=_between(rng, 40, 160), rho=1.2, jitter=0.1, precision="mixed",
                     skin=rng.choice((0.3, 0.4)), pinned=True, energy=rng.random() < 0.3)
    return _case(mode="run", lattice="mix", m=_between(rng, 48, 200), rho=1.2, jitter=0.1, precision="mixed",
                 skin=rng.choice((0.3, 0.4)), tile=rng.choice((0, 5)), steps=21, dt=0.003)


# ---- inputs -----------------------------------------------------------------
_FCC = ((0.0, 0.0, 0.0), (0.5, 0.5, 0.0), (0.5, 0.0, 0.5), (0.0, 0.5, 0.5))
_SC = ((0.5, 0.5, 0.5),)
MOVE = 0.02  # of the lattice spacing: how far a call's atoms are from where its context began, per coordinate


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _grid(n, a, basis, jitter, gen, lo=(0.0, 0.0, 0.0)):
    """Sites of an n[0] x n[1] x n[2] lattice with spacings a, each coordinate moved by up to jitter * a."""
    dev = gen.device
    k, j, i = torch.meshgrid(*(torch.arange(n[t], device=dev) for t in (2, 1, 0)), indexing="ij")
    cell = torch.stack([i.reshape(-1), j.reshape(-1), k.reshape(-1)], 1).to(torch.float64)
    p = (cell[:, None, :] + torch.tensor(basis, dtype=torch.float64, device=dev)[None]).reshape(-1, 3)
    p += jitter * (2.0 * torch.rand(p.shape, dtype=torch.float64, device=dev, generator=gen) - 1.0)
    return p * torch.tensor(a, dtype=torch.float64, device=dev) + torch.tensor(lo, dtype=torch.float64, device=dev)


def _gen(seed):
    gen = torch.Generator(device=_device())
    gen.manual_seed(int(seed))
    return gen


def _sites(case, gen, jit):
    """Positions of the case's lattice, each coordinate moved by up to jit of the spacing; box edges, atoms per box."""
    m, rho = case["m"], case["rho"]
    if case["lattice"] == "fcc":
        a = (4.0 / rho) ** (1.0 / 3.0)
        parts, boxes = [_grid((m, m, m), (a, a, a), _FCC, jit, gen)], [(m * a,) * 3]
    elif case["lattice"] in ("sc", "mix"):
        a = (1.0 / rho) ** (1.0 / 3.0)
        parts, boxes = [_grid((m, m, m), (a, a, a), _SC, jit, gen)], [(m * a,) * 3]
    elif case["lattice"] == "slab":
        lx = m / rho ** (1.0 / 3.0)  # the liquid: a cube of m^3 sites in the middle quarter of z
        a, v = lx / m, (1.0 / 0.02) ** (1.0 / 3.0)
        nv = (int(round(lx / v)), int(round(lx / v)), int(round(1.5 * lx / v)))
        av = (lx / nv[0], lx / nv[1], 1.5 * lx / nv[2])
        parts = [torch.cat([_grid((m, m, m), (a, a, a), _SC, jit, gen, (0.0, 0.0, 1.5 * lx)),
                            _grid(nv, av, _SC, 0.3, gen), _grid(nv, av, _SC, 0.3, gen, (0.0, 0.0, 2.5 * lx))])]
        boxes = [(lx, lx, 4.0 * lx)]
    else:  # ensemble: atoms log-uniform in [256, 16384], density 0.3 to 0.9; the boxes belong to the case
        r = np.random.default_rng(case["boxes"])
        parts, boxes = [], []
        for _ in range(case["boxes"]):
            n = math.exp(r.uniform(math.log(256), math.log(16384)))
            d = r.uniform(0.3, 0.9)
            if r.random() < 0.5:
                k, a, basis = max(4, int(round((n / 4) ** (1 / 3)))), (4.0 / d) ** (1.0 / 3.0), _FCC
            else:
                k, a, basis = max(7, int(round(n ** (1 / 3)))), (1.0 / d) ** (1.0 / 3.0), _SC
            parts.append(_grid((k, k, k), (a, a, a), basis, jit, gen))
            boxes.append((k * a,) * 3)
    return torch.cat(parts), boxes, [len(p) for p in parts]


def _wrapped(pos, L):
    pos = pos.remainder(L)
    return torch.where(pos >= L, torch.zeros((), dtype=pos.dtype, device=pos.device), pos)


def _atoms(case, seed):
    """Positions, velocities, types (or None), box edges (nboxes, 3), atoms per box and box of an atom, made from the
    seed; the positions of a call are near those that the context began with (_begin)."""
    gen = _gen(seed)
    if case["mode"] == "call":
        pos, boxes, counts = _sites(case, _gen(0), case["jitter"] - MOVE)
        a = (4.0 if case["lattice"] == "fcc" else 1.0) / case["rho"]
        pos += MOVE * a ** (1.0 / 3.0) * (2.0 * torch.rand(pos.shape, dtype=pos.dtype, device=pos.device,
                                                           generator=gen) - 1.0)
    else:
        pos, boxes, counts = _sites(case, gen, case["jitter"])
    dev = pos.device
    L = torch.tensor(boxes, dtype=torch.float64, device=dev)
    box = torch.repeat_interleave(torch.arange(len(counts), device=dev), torch.tensor(counts, device=dev))
    pos = _wrapped(pos, L[box])
    types = None
    if case["lattice"] == "mix":
        types = (torch.rand(len(pos), device=dev, generator=_gen(1)) < 0.2).to(torch.int32)
    if case["mode"] != "run":
        return pos, None, types, boxes, counts, box
    # Maxwell-Boltzmann velocities, zero net momentum, the kinetic temperature exact in every box
    # (an ensemble's temperatures: 0.7 to 1.5)
    temps = [case["temp"]] if len(counts) == 1 else np.random.default_rng(len(counts)).uniform(0.7, 1.5, len(counts))
    vel = torch.randn(pos.shape, dtype=torch.float64, device=dev, generator=gen)
    nb = torch.tensor(counts, dtype=torch.float64, device=dev)
    vel -= (torch.stack([torch.bincount(box, vel[:, c], len(counts)) for c in range(3)], 1) / nb[:, None])[box]
    ke2 = torch.bincount(box, (vel * vel).sum(1), len(counts))
    T = torch.as_tensor(temps, dtype=torch.float64, device=dev)
    vel *= torch.sqrt(3.0 * (nb - 1.0) * T / ke2)[box][:, None]
    return pos, vel, types, boxes, counts, box


def _begin(case):
    """The positions that a call's context began with."""
    pos, boxes, _ = _sites(case, _gen(0), case["jitter"] - MOVE)
    return _wrapped(pos, torch.tensor(boxes[0], dtype=torch.float64, device=pos.device)).cpu().numpy()


def _lj(case):
    if case["lattice"] != "mix":
        return {"rc": case["rc"]}
    return {"ntypes": 2, "eps": MIX_EPS, "sigma": MIX_SIGMA, "rc": (case["rc"] * np.array(MIX_SIGMA)).tolist()}


_kept = {}  # the context of the runs of one case, kept from one configuration to the next as a program keeps it


def _system(case, boxes, counts):
    kw = dict(_lj(case), precision=case["precision"], potential=case["potential"], pair_skin=case["skin"],
              tile_balance=case["balance"])
    if case["tile"]:
        kw["tile"] = case["tile"]
    return ex.MidpointLJ(boxes, counts, **kw)


def _host(t, pinned):
    a = t.cpu().numpy()
    if not pinned:
        return a
    p = ex.pinned_empty(a.shape)
    p[:] = a
    return p


def prepare(case, seed):
    pos, vel, types, boxes, counts, _ = _atoms(case, seed)
    types = None if types is None else types.cpu().numpy()
    if case["mode"] == "oneshot":
        return {"case": case, "pos": pos.cpu().numpy(), "boxes": boxes}
    pinned = case["pinned"] or case["mode"] == "run"
    st = {"case": case, "pos": _host(pos, pinned), "types": types}
    if case["out"] == "forces":
        st["forces"] = (ex.pinned_empty if pinned else np.empty)(tuple(pos.shape))
    if case["mode"] == "call":
        st["system"] = _system(case, boxes, counts)
        st["system"].set_atoms(_begin(case), types)
        return st
    st["vel"] = _host(vel, True)
    key = tuple(sorted(case.items()))
    if key not in _kept:
        for k in list(_kept):
            _kept.pop(k).close()
        _kept[key] = _system(case, boxes, counts)
        _kept[key].set_atoms(st["pos"], types, st["vel"])
        _kept[key].prepare_run(case["dt"], CHUNK, energies=case["energy"])
    st["system"] = _kept[key]
    return st


def run(state):
    case = state["case"]
    if case["mode"] == "oneshot":
        f, epot, virial = ex.forces_midpoint_all(state["pos"], state["boxes"][0], case["rc"],
                                                 precision=case["precision"], energy=True)
        return {"forces": f, "epot": epot, "virial": virial}
    s = state["system"]
    if case["mode"] == "call":
        f = state["forces"]
        if case["accumulate"]:
            f.fill(0.0)
        f, epot, virial = s.forces_at(state["pos"], out=f, accumulate=case["accumulate"], energy=case["energy"])
        return {"forces": f, "epot": epot, "virial": virial} if case["energy"] else {"forces": f}
    s.set_atoms(state["pos"], state["types"], state["vel"])
    r = s.run(case["steps"], case["dt"], graph_chunk=CHUNK, energies=case["energy"])
    out = {"ekin": r["ekin"], "epot": r["epot"]} if case["energy"] else {}
    if case["out"] == "state":
        out["pos"], out["vel"] = s.state()
    else:
        out["forces"] = s.forces(out=state["forces"])[0]
    return out


# ---- work and exact values --------------------------------------------------
def _sizes(case):
    """(atoms, pairs within the cutoff) of a case, from its lattice and mean density."""
    m, third = case["m"], 2.0 * math.pi / 3.0
    if case["lattice"] == "ensemble":  # the means of the sizes and densities drawn
        n = int(case["boxes"] * (16384 - 256) / math.log(64.0))
        return n, n * 0.6 * third * case["rc"] ** 3
    if case["lattice"] == "slab":
        lx = m / case["rho"] ** (1.0 / 3.0)
        return int(m ** 3 + 0.06 * lx ** 3), (m ** 3 * case["rho"] + 0.06 * lx ** 3 * 0.02) * third * case["rc"] ** 3
    n = 4 * m ** 3 if case["lattice"] == "fcc" else m ** 3
    vol = case["rc"] ** 3
    if case["lattice"] == "mix":  # cutoff rc sigma_ab, 80:20
        vol *= sum(x * y * MIX_SIGMA[a][b] ** 3 for a, x in enumerate((0.8, 0.2)) for b, y in enumerate((0.8, 0.2)))
    return n, n * case["rho"] * third * vol


def work(case):
    # 30 operations a pair within the cutoff (distance 8, force and both sums 22), 18 an atom and step of a run
    n, pairs = _sizes(case)
    evals = case["steps"] + (case["out"] == "forces") if case["mode"] == "run" else 1
    flops = evals * 30.0 * pairs + 18.0 * n * case["steps"]
    nbytes = 48.0 * n  # positions in and forces out
    if case["mode"] == "run":  # positions and velocities in and out, or the forces out
        nbytes = (96.0 if case["out"] == "state" else 72.0) * n
    return {"bytes": nbytes, "flops": flops}


class _Pairs:
    """Forces and energies in 64 bits by a list of all pairs within the cutoff and a margin."""

    def __init__(self, case, types, boxes, counts, box):
        self.dev, self.box, self.nbox = box.device, box, len(counts)
        self.L = torch.tensor(boxes, dtype=torch.float64, device=self.dev)
        lj = _lj(case)
        t = lambda v: torch.tensor(v, dtype=torch.float64, device=self.dev).reshape(-1)  # noqa: E731
        self.nt = lj.get("ntypes", 1)
        self.eps, self.sig, self.rc = t(lj.get("eps", 1.0)), t(lj.get("sigma", 1.0)), t(lj["rc"])
        self.types, self.margin, self.at = types, 0.3 if case["mode"] == "run" else 0.0, None
        self.cut2, self.shift = self.rc ** 2, torch.zeros_like(self.rc)
        s6 = (self.sig / self.rc) ** 6
        if case["potential"] == "lj_shifted":
            self.shift = 4.0 * self.eps * s6 * (s6 - 1.0)
        elif case["potential"] == "wca":
            self.cut2, self.shift = 2.0 ** (1.0 / 3.0) * self.sig ** 2, -self.eps

    def _image(self, d, k):
        L = self.L[0] if self.nbox == 1 else self.L[self.box[k]]
        return d - L * torch.round(d / L)

    def _build(self, x):
        reach = float(self.rc.max()) + self.margin
        nc = torch.clamp(torch.floor(self.L / reach), 1, 1023).to(torch.int64)  # cells per box and axis
        first = torch.cumsum(nc.prod(1), 0) - nc.prod(1)
        n = nc[self.box]
        c = torch.minimum((x / self.L[self.box] * n).to(torch.int64), n - 1)
        cell = lambda q: first[self.box] + q[:, 0] + n[:, 0] * (q[:, 1] + n[:, 1] * q[:, 2])  # noqa: E731
        order = torch.argsort(cell(c))
        rank = torch.empty_like(order)
        rank[order] = torch.arange(len(order), device=self.dev)
        size = torch.bincount(cell(c), minlength=int(nc.prod(1).sum()))
        start = torch.cumsum(size, 0) - size
        most, got = int(size.max()), []
        for o in range(27):
            off = torch.tensor((o % 3 - 1, o // 3 % 3 - 1, o // 9 - 1), device=self.dev)
            # fewer than 3 cells on an axis: each neighbour once
            ok = (((off == 0) | (n >= 3) | ((off == 1) & (n == 2))).all(1))
            q = cell((c + off).remainder(n))
            b, e = start[q], size[q]
            for k in range(most):
                i = torch.nonzero(ok & (k < e) & (b + k > rank)).reshape(-1)
                j = order[b[i] + k]
                near = (self._image(x[j] - x[i], i) ** 2).sum(1) <= reach * reach
                got.append((i[near].to(torch.int32), j[near].to(torch.int32)))
        self.i, self.j = torch.cat([g[0] for g in got]), torch.cat([g[1] for g in got])
        self.at = x.clone()

    def forces(self, x):
        if self.at is None or float((self._image(x - self.at, slice(None)) ** 2).sum(1).max()) > (self.margin / 2) ** 2:
            self._build(x)
        f = torch.zeros_like(x)
        epot, vir = (torch.zeros(self.nbox, dtype=torch.float64, device=self.dev) for _ in range(2))
        for lo in range(0, len(self.i), 1 << 26):
            i, j = self.i[lo:lo + (1 << 26)].long(), self.j[lo:lo + (1 << 26)].long()
            d = self._image(x[j] - x[i], i)
            r2 = (d * d).sum(1)
            p = torch.zeros_like(i) if self.types is None else (self.types[i] * self.nt + self.types[j]).long()
            use = (r2 <= self.rc[p] ** 2) & (r2 <= self.cut2[p])
            i, j, d, r2, p = i[use], j[use], d[use], r2[use], p[use]
            s6 = (self.sig[p] ** 2 / r2) ** 3
            dg = -24.0 * self.eps[p] * (2.0 * s6 * s6 - s6) / r2
            f.index_add_(0, i, dg[:, None] * d)
            f.index_add_(0, j, -dg[:, None] * d)
            b = self.box[i]
            epot += torch.bincount(b, 4.0 * self.eps[p] * (s6 * s6 - s6) - self.shift[p], self.nbox)
            vir += torch.bincount(b, -dg * r2, self.nbox)
        return f, epot, vir


def exact(case, seed):
    n, pairs = _sizes(case)
    evals = 1 + case["steps"]
    if pairs * evals > 4e9:  # over about 20 seconds
        return None
    x, v, types, boxes, counts, box = _atoms(case, seed)
    P = _Pairs(case, types, boxes, counts, box)
    f, epot, vir = P.forces(x)
    host = lambda t: t.cpu().numpy()  # noqa: E731
    if case["mode"] != "run":
        if case["mode"] == "oneshot":
            return {"forces": host(f), "epot": float(epot[0]), "virial": float(vir[0])}
        return {"forces": host(f), "epot": host(epot), "virial": host(vir)} if case["energy"] else {"forces": host(f)}
    L, h, ek, ep = P.L[box], 0.5 * case["dt"], [], []
    for _ in range(case["steps"]):  # velocity-Verlet, unit masses
        v = v + h * f
        x = _wrapped(x + case["dt"] * v, L)
        f, epot, _ = P.forces(x)
        v = v + h * f
        ek.append(torch.bincount(box, 0.5 * (v * v).sum(1), len(counts)))
        ep.append(epot)
    out = {"ekin": host(torch.stack(ek)), "epot": host(torch.stack(ep))} if case["energy"] else {}
    if case["out"] == "state":
        out["pos"], out["vel"] = host(x), host(v)
    else:
        out["forces"] = host(f)
    return out
