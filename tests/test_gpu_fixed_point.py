"""The FP64 form's fixed-point first pass, the order of the pair lists, and the
energies of runs.

- The fixed-point pass (positions, r^2 and force sums as integers) gives the
  oracle's forces within the FP64 form's 1e-12 of F_rms, energy and virial, and
  the same pair counts: for boxes around powers of two (where a separation
  across the periodic face is rounded at another bit), small and elongated
  ones, other units of length and energy, and several types.
- Tiles it cannot compute go to the FP64 body: forces beyond the sums' range,
  tiles over the first pass's capacity, and every tile where the type pairs'
  force scales differ too much for one unit.
- A list's entries are put in another order in groups of 32: lists shorter and
  longer than a group, and the types carried by the entries, against the
  enumeration at the build, bit for bit.
- A run's energies do not depend on how its steps are grouped into graphs and
  copies.
"""
import numpy as np
import pytest

pytestmark = [pytest.mark.gpu]

TOL64 = 1e-12
KA = dict(ntypes=2, eps=[[1.0, 1.5], [1.5, 0.5]], sigma=[[1.0, 0.8], [0.8, 0.88]], rc=[[2.5, 2.0], [2.0, 2.2]])


def frms(f):
    return np.sqrt((f * f).sum(1).mean())


def edge(rc):
    """The library's cell edge: rc / 2 rounded up to 14 significant bits."""
    h = 0.5 * np.max(rc)
    unit = 2.0 ** (np.floor(np.log2(h)) - 13)
    return float(np.ceil(h / unit) * unit)


def against_oracle(gpulib, oracle, pos, L, types=None, **lj):
    ref = oracle.forces_typed(pos, L, lj["rc"], types=types, threads=0, block_length=edge(lj["rc"]),
                              **{k: v for k, v in lj.items() if k in ("eps", "sigma", "ntypes")})
    with gpulib.MidpointLJ(L, [len(pos)], precision="fp64", **lj) as s:
        s.set_atoms(pos, types)
        f, e, w = s.forces(energy=True)
        plain, _, _ = s.forces()
        cnt = s.counters()
    fr = ref["forces"]
    for g in (f, plain):
        assert np.sqrt(((g - fr) ** 2).sum(1)).max() <= TOL64 * frms(fr)
    assert e[0] == pytest.approx(ref["epot"], rel=TOL64) and w[0] == pytest.approx(ref["virial"], rel=TOL64)
    assert cnt["candidates"] == ref["counts"].candidates and cnt["accepted"] == ref["counts"].accepted


@pytest.mark.parametrize("L,n", [((7.999, 8.0, 8.001), 300), ((16.0, 15.9999, 33.0), 5000), ((6.3, 6.3, 64.0), 1500),
                                 ((12.6, 12.6, 12.6), 1)])
def test_boxes(gpulib, oracle, L, n):
    L = np.array(L)
    pos = gpulib.gen_random(n, L, 0.8, 7)
    # a third of the atoms next to a face, on either side, down to the smallest doubles
    rng = np.random.default_rng(3)
    if n > 1:
        k = rng.integers(0, n, n // 3)
        near = np.array([0.0, 1e-300, 1e-17, 3e-9, 1e-4])[rng.integers(0, 5, len(k))]
        a = rng.integers(0, 3, len(k))
        moved = pos.copy()
        moved[k, a] = np.where(rng.random(len(k)) < 0.5, near, np.nextafter(L[a], 0.0) - near)
        from scipy.spatial import cKDTree
        close = cKDTree(moved, boxsize=L).query_pairs(0.75, output_type="ndarray")
        keep = np.ones(n, dtype=bool)
        keep[close[:, 1]] = False
        pos = np.ascontiguousarray(moved[keep])
    if n == 1:
        with gpulib.MidpointLJ(L, [1], precision="fp64") as s:
            s.set_atoms(pos)
            assert not s.forces()[0].any()
        return
    against_oracle(gpulib, oracle, pos, L, rc=2.5)


@pytest.mark.parametrize("eps,sigma", [(0.0103, 3.405), (250.0, 0.02), (1.0, 1.7)])
def test_units(gpulib, oracle, eps, sigma):
    L = np.array([13.0, 14.0, 15.0])
    pos = gpulib.gen_random(2000, L, 0.8, 11) * sigma
    against_oracle(gpulib, oracle, np.ascontiguousarray(pos), L * sigma, rc=2.5 * sigma, eps=eps, sigma=sigma)


@pytest.mark.parametrize("lj", [KA, dict(KA, eps=[[1.0, 0.3], [0.3, 0.0625]]), dict(KA, eps=[[1.0, 0.1], [0.1, 0.01]]),
                                dict(ntypes=1, eps=1.0, sigma=1.0, rc=0.7)])
def test_types(gpulib, oracle, lj):
    """Force scales within and beyond a factor of 16 of each other (the last two cases have no fixed-point pass)."""
    L = np.array([11.0, 12.0, 13.0])
    pos = gpulib.gen_random(1500, L, 0.6 if lj["ntypes"] == 1 else 0.85, 5)
    types = None if lj["ntypes"] == 1 else (np.random.default_rng(1).random(1500) < 0.3).astype(np.int32)
    against_oracle(gpulib, oracle, pos, L, types, **lj)


def test_forces_beyond_the_sums(gpulib, oracle):
    """Pairs down to 0.5 sigma (|F| to 4e5) in some tiles, none in others."""
    L = np.array([14.0, 15.0, 30.0])
    pos = gpulib.gen_random(4000, L, 0.85, 9)
    rng = np.random.default_rng(2)
    for i in range(0, 200, 2):
        pos[i + 1] = pos[i] + rng.uniform(0.5, 0.72) * np.array([0.6, 0.48, 0.64])
    low = (pos % L)[:, 2] < 12.0
    pos = np.ascontiguousarray((pos % L)[low | (np.arange(4000) >= 200)])
    against_oracle(gpulib, oracle, pos, L, rc=2.5)


@pytest.mark.parametrize("neighbours", [1, 2, 4])
def test_several_large_terms_on_one_atom(gpulib, oracle, neighbours):
    """Atoms with 1, 2 or 4 neighbours at 0.745 to 0.83 sigma on one side, every term within the first pass's range
    (|F| 500 to 2000); four of them add up to nearly what the sums hold (4096)."""
    rng = np.random.default_rng(neighbours)
    L = np.array([16.0, 20.0, 24.0])
    c = np.stack(np.meshgrid(*[np.arange(1.0, b, 4.0) for b in L], indexing="ij"), -1).reshape(-1, 3)
    t = np.radians(50.0)
    parts = [c]
    for k in range(neighbours):
        u = np.array([np.cos(t), np.sin(t) * np.cos(k * np.pi / 2), np.sin(t) * np.sin(k * np.pi / 2)])
        parts.append(c + rng.uniform(0.745, 0.83, (len(c), 1)) * u)
    against_oracle(gpulib, oracle, np.concatenate(parts), L, rc=2.5)


def test_first_pass_overflow(gpulib, oracle):
    """A density wave through forces_at packs tiles beyond the first pass's capacity (6 % + 32 atoms above the
    largest tile when the atoms were set), within the redo pass's (25 % + 64)."""
    from examd_gb300 import workloads as W
    c = W.liquid_fcc(16)
    L, pos = np.asarray(c["boxes"][0]), c["pos"]

    def squeeze(a):
        p = pos.copy()
        p[:, 2] = (pos[:, 2] - a * L[2] / (2 * np.pi) * np.sin(2 * np.pi * pos[:, 2] / L[2])) % L[2]
        return p

    def largest(p):
        with gpulib.MidpointLJ(L, [len(p)], precision="fp64") as s:
            s.set_atoms(p)
            return s.counters()["max_tile_atoms"]

    occ = largest(pos)
    first, redo = (occ + occ // 16 + 32 + 7) // 8 * 8, (occ + occ // 4 + 64 + 7) // 8 * 8
    new = next(squeeze(a) for a in (0.25, 0.3, 0.35, 0.4, 0.45, 0.5) if first < largest(squeeze(a)) <= redo)
    with gpulib.MidpointLJ(L, [len(pos)], precision="fp64") as s:
        s.set_atoms(pos)
        f, e, _ = s.forces_at(new, energy=True)
    ref = oracle.forces_typed(new, L, 2.5, threads=0)
    assert np.sqrt(((f - ref["forces"]) ** 2).sum(1)).max() <= TOL64 * frms(ref["forces"])
    assert e[0] == pytest.approx(ref["epot"], rel=TOL64)


def test_two_contexts_side_by_side(gpulib):
    """A second context of smaller tiles does not take shared memory away from the first."""
    from examd_gb300 import workloads as W
    c = W.liquid_fcc(12)
    out = []
    with gpulib.MidpointLJ(c["boxes"], c["natoms"], precision="fp64", tile=6) as a:
        a.set_atoms(c["pos"])
        out.append(a.forces()[0])
        with gpulib.MidpointLJ(c["boxes"], c["natoms"], precision="fp64", tile=2) as b:
            b.set_atoms(c["pos"])
            b.forces()
            out.append(a.forces()[0])
    assert np.array_equal(out[0], out[1])


@pytest.mark.parametrize("rc,skin,ntypes", [(1.2, 0.1, 1), (2.5, 0.4, 4), (3.5, 0.5, 1), (3.0, 0.3, 2)])
def test_list_order(gpulib, rc, skin, ntypes):
    """Lists of a few to about 150 entries (several groups of 32), one to four types."""
    from examd_gb300 import workloads as W
    c = W.liquid_fcc(12)
    t = None if ntypes == 1 else np.random.default_rng(4).integers(0, ntypes, len(c["pos"])).astype(np.int32)
    k = np.arange(ntypes)
    scale = 1.0 - 0.05 * (k[:, None] + k[None, :])
    out = []
    for s_ in (0.0, skin):
        with gpulib.MidpointLJ(c["boxes"], c["natoms"], precision="mixed", rc=rc * scale, sigma=scale, eps=1.0 / scale,
                               ntypes=ntypes, block_length=0.5 * (rc + skin), pair_skin=s_) as s:
            s.set_atoms(c["pos"], t)
            out.append(s.forces(energy=True))
            if s_:
                info = s.list_info()
                assert info["fallback_tiles"] == 0
    for x, y in zip(*out):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("skin", [0.0, 0.3])
def test_energies_of_grouped_steps(gpulib, skin):
    """45 steps of three boxes: eager (more steps than are held on the device), graphs of 4 and of 20 steps."""
    from examd_gb300 import workloads as W
    c = [W.liquid_fcc(k, seed=k) for k in (6, 7, 8)]
    pos, vel = (np.concatenate([x[n] for x in c]) for n in ("pos", "vel"))
    boxes, counts = np.concatenate([x["boxes"] for x in c]), np.concatenate([x["natoms"] for x in c])
    out = []
    for chunk in (0, 4, 20):
        with gpulib.MidpointLJ(boxes, counts, precision="mixed", pair_skin=skin) as s:
            s.set_atoms(pos, vel=vel)
            r = s.run(45, 0.004, graph_chunk=chunk, energies=True)
            last = s.forces(energy=True)[1]
            out.append((r["ekin"], r["epot"], s.kinetic(), last))
    for o in out:
        assert o[0].shape == (45, 3) and np.allclose(o[0][-1], o[2], rtol=1e-12) and np.allclose(o[1][-1], o[3], rtol=1e-12)
        if skin == 0.0:  # (with lists the rebuilds fall alike unless a capacity grows between graphs)
            # the potential energies are exact sums; the kinetic ones are FP64 sums over the sorted atoms, whose
            # order inside a cell is not fixed: at most n 2^-53 apart
            assert np.array_equal(o[1], out[0][1])
            assert np.allclose(o[0], out[0][0], rtol=2.0 ** -53 * counts.max(), atol=0.0)
        assert np.allclose(o[0], out[0][0], rtol=1e-6) and np.allclose(o[1], out[0][1], rtol=1e-6)
