"""The range and the resolution of the FP64 form's fixed-point pass.

- Any number of terms on one atom: many small neighbours on one side of a large
  atom, and a cluster whose own pairs another tile computes.
- Weak pairs keep FP64's relative accuracy: isolated pairs near the cutoff, at
  cutoffs of 2.5 to 8 sigma, of the weakest type pair beside a strong one, and
  contact pairs far inside the largest cutoff.  The bound is that of the FP64
  body's own expression, in units of u = 2^-53: each separation is rounded once
  (1 u), r^2 5 u, 1 / r^2 6 u, sigma^2 / r^2 8 u, its cube 26 u, squared 53 u, the
  difference, eps, 1 / r^2 and the separation 12 u more: 65 u of the repulsive
  and 38 u of the attractive term.
"""
import numpy as np
import pytest

pytestmark = [pytest.mark.gpu]

TOL64 = 1e-12
U = 2.0 ** -53


def lj_exact(pos, pairs, eps, sigma):
    """Forces of the listed pairs from the exact difference of their coordinates (no periodic images), in extended
    precision, and the bound of the FP64 expression's error."""
    q = np.longdouble
    d = pos.astype(q)[pairs[:, 1]] - pos.astype(q)[pairs[:, 0]]
    r2 = (d * d).sum(1)
    s6 = (q(sigma) * q(sigma) / r2) ** 3
    dg = -24 * q(eps) * (2 * s6 * s6 - s6) / r2
    size = 24 * q(eps) / np.sqrt(r2) * (2 * s6 * s6 * 65 + s6 * 38) * U
    return dg[:, None] * d, size


def directions(k, rng):
    u = rng.normal(size=(k, 3))
    return u / np.sqrt((u * u).sum(1))[:, None]


@pytest.mark.parametrize("sigma_b,count,angle", [(0.2, 27, 60.0), (0.45, 15, 78.0), (0.45, 9, 60.0)])
def test_many_small_neighbours_on_one_side(gpulib, oracle, sigma_b, count, angle):
    """Atoms of type 0 with `count` atoms of type 1 on a cap of 0.826 sigma around each, every term below 2^9 but
    their sum twice 4096 or so; the small ones beyond their own potential's minimum from each other."""
    L = np.array([18.0, 24.0, 30.0])
    c = np.stack(np.meshgrid(*[np.arange(3.0, b, 6.0) for b in L], indexing="ij"), -1).reshape(-1, 3)
    # spiral points on the cap, evenly spread
    k = np.arange(count) + 0.5
    z = 1.0 - (1.0 - np.cos(np.radians(angle))) * k / count
    phi = np.pi * (1.0 + 5.0 ** 0.5) * k
    u = np.stack([z, np.sqrt(1 - z * z) * np.cos(phi), np.sqrt(1 - z * z) * np.sin(phi)], 1)
    parts, types = [c], [np.zeros(len(c), dtype=np.int32)]
    for v in 0.826 * u:
        parts.append(c + v)
        types.append(np.ones(len(c), dtype=np.int32))
    pos, types = np.concatenate(parts), np.concatenate(types)
    lj = dict(ntypes=2, eps=[[1.0, 1.0], [1.0, sigma_b]], sigma=[[1.0, 1.0], [1.0, sigma_b]],
              rc=[[2.5, 2.5], [2.5, 2.5 * sigma_b]])
    ref = oracle.forces_typed(pos, L, lj["rc"], types=types, threads=0, block_length=1.25,
                              **{k: lj[k] for k in ("eps", "sigma", "ntypes")})
    with gpulib.MidpointLJ(L, [len(pos)], precision="fp64", **lj) as s:
        s.set_atoms(pos, types)
        f, e, _ = s.forces(energy=True)
    fr = ref["forces"]
    assert np.abs(fr[:len(c), 0]).min() > (4096 if count > 9 else 2000)
    assert np.sqrt(((f - fr) ** 2).sum(1)).max() <= TOL64 * np.sqrt((fr * fr).sum(1).mean())
    assert e[0] == pytest.approx(ref["epot"], rel=TOL64)


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("side", [-1.0, 1.0])
def test_cluster_in_the_next_tile(gpulib, axis, side):
    """16 atoms within 0.01 of each other, 0.84 sigma from a single atom across each tile face of the axis: the tile
    of the cluster's own pairs may not be the one that sums the single atom's."""
    L = np.full(3, 30.0)
    rng = np.random.default_rng(1)
    singles, clusters = [], []
    for t in (2, 3, 4):  # tiles of t cells of 1.25 on every axis
        for k in range(1, int(24 / t)):
            x = np.full(3, 5.0)
            x[(axis + 1) % 3] += 2.6 * (k % 8)
            x[(axis + 2) % 3] += 2.6 * (k // 8) + 7.8 * (t - 2)
            x[axis] = 1.25 * t * k - side * 0.42
            y = x.copy()
            y[axis] += side * 0.84
            if all(np.abs(x - z).max() > 4.5 for z in singles):
                singles.append(x)
                clusters.append(y + rng.uniform(-0.005, 0.005, (16, 3)))
    pos = np.concatenate([np.array(singles)] + clusters)
    n = len(singles)
    assert n >= 3
    for tile in (2, 3, 4):
        with gpulib.MidpointLJ(L, [len(pos)], precision="fp64", tile=tile) as s:
            s.set_atoms(pos)
            f = s.forces()[0]
        for i in range(n):
            k = n + 16 * i + np.arange(16)
            F, size = lj_exact(pos, np.stack([np.full(16, i), k], 1), 1.0, 1.0)
            # the exact terms' sum, their own error and that of 16 FP64 additions
            assert np.abs(f[i] - F.sum(0)).max() <= float(size.sum()) + 16 * U * float(np.abs(F).sum())


@pytest.mark.parametrize("rc", [2.5, 3.0, 3.8, 4.0, 5.0, 6.0, 8.0])
@pytest.mark.parametrize("what", ["cutoff", "middle", "contact", "weak"])
def test_isolated_pairs(gpulib, rc, what):
    """weak: the type pair of a sixteenth of the strongest one's eps."""
    m = 7
    spacing = 2.2 * rc
    L = np.full(3, m * spacing)
    rng = np.random.default_rng(int(10 * rc))
    c = (np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3) + 0.5) * spacing
    lo, hi = {"cutoff": (0.95 * rc, 0.999 * rc), "middle": (1.5, 2.4), "contact": (0.9, 1.05),
              "weak": (0.8 * rc, 0.999 * rc)}[what]
    half = 0.5 * rng.uniform(lo, hi, len(c))[:, None] * directions(len(c), rng)
    pos = np.concatenate([c - half, c + half])
    pairs = np.stack([np.arange(len(c)), np.arange(len(c)) + len(c)], 1)
    if what == "weak":
        lj, types, eps = dict(ntypes=2, eps=[[1.0, 0.25], [0.25, 0.0625]], rc=rc), np.ones(len(pos), dtype=np.int32), 0.0625
    else:
        lj, types, eps = dict(rc=rc), None, 1.0
    F, size = lj_exact(pos, pairs, eps, 1.0)
    with gpulib.MidpointLJ(L, [len(pos)], precision="fp64", **lj) as s:
        s.set_atoms(pos, types)
        f = s.forces()[0]
        assert s.counters()["accepted"] == len(c)
    n = len(c)
    for sign, g in ((1, f[:n]), (-1, f[n:])):
        err = np.sqrt(((sign * g - F) ** 2).sum(1)).astype(np.float64)
        assert (err <= size.astype(np.float64)).all(), float((err / size).max())


@pytest.mark.parametrize("ratio", [1.0, 2.0, 3.0, 4.0, 8.0, 15.0])
def test_small_pairs_beside_a_long_cutoff(gpulib, ratio):
    """Contact pairs of a type `ratio` times smaller than the one whose cutoff is the longest: the RMS error is no
    larger than that of FP64's own expression on the same pairs.  Of 1,000 pairs each RMS is known to about 5 %
    (errors between uniform and normal), so the quotient to 7 %: three of that, 1.2."""
    m, s = 10, 1.0 / ratio
    rc = np.array([[2.5, 1.25 * (1 + s)], [1.25 * (1 + s), 2.5 * s]])
    L = np.full(3, m * 1.6)
    rng = np.random.default_rng(int(ratio))
    c = (np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3) + 0.5) * 1.6
    c = c if ratio > 1.0 else c * 2.5
    L = L if ratio > 1.0 else L * 2.5
    spread = 2.2 * 2.5 * s  # the small pairs' own cutoff is what separates them
    if ratio > 1.0 and spread > 1.6:
        c, L = c * (spread / 1.6), L * (spread / 1.6)
    half = 0.5 * s * rng.uniform(0.9, 1.05, len(c))[:, None] * directions(len(c), rng)
    pos = np.concatenate([c - half, c + half])
    n = len(c)
    pairs = np.stack([np.arange(n), np.arange(n) + n], 1)
    lj = dict(ntypes=2, eps=1.0, sigma=[[1.0, 0.5 * (1 + s)], [0.5 * (1 + s), s]], rc=rc)
    F, _ = lj_exact(pos, pairs, 1.0, s)
    with gpulib.MidpointLJ(L, [len(pos)], precision="fp64", **lj) as sysm:
        sysm.set_atoms(pos, np.ones(len(pos), dtype=np.int32))
        f = sysm.forces()[0]
        assert sysm.counters()["accepted"] == n
    d = pos[n:] - pos[:n]
    r2 = d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1] + d[:, 2] * d[:, 2]
    i2 = 1.0 / r2
    t = (s * s) * i2
    d6 = t * t * t
    f64 = (-(24.0 * (2.0 * (d6 * d6) - d6)) * i2)[:, None] * d
    size = np.sqrt((F * F).sum(1))

    def rms(g):
        return float(np.sqrt((((g - F) ** 2).sum(1) / size ** 2).mean()))

    assert rms(f[:n]) <= 1.2 * rms(f64) and rms(-f[n:]) <= 1.2 * rms(f64)


@pytest.mark.parametrize("potential,m,rho,jitter,rc", [("wca", 16, 1.05, 0.0001, 2.5), ("wca", 16, 1.0, 0.02, 2.5),
                                                      ("lj_shifted", 12, 0.95, 0.03, 1.6), ("lj", 14, 0.8442, 0.09, 2.5)])
def test_energy_and_virial_to_fp64(gpulib, potential, m, rho, jitter, rc):
    """Energies near a potential's end and sums over many pairs: the RMS error over eight configurations is the pairs'
    own in FP64 (independent, as the FP64 expression has them) and the rounding of the last few sums, 0.41 u."""
    from scipy.spatial import cKDTree
    q = np.longdouble
    a = (4.0 / rho) ** (1.0 / 3.0)
    L = np.full(3, m * a)
    basis = np.array([[0, 0, 0], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]])
    g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 1, 3)
    shift = {"lj": q(0), "wca": q(-1), "lj_shifted": 4 * (1 / q(rc) ** 12 - 1 / q(rc) ** 6)}[potential]
    rel, allow = [], 0.0
    for seed in range(8):
        rng = np.random.default_rng(seed)
        x = ((g + basis).reshape(-1, 3) + 0.25 + jitter * rng.uniform(-1, 1, (4 * m ** 3, 3))) * a % L
        p = cKDTree(x, boxsize=L).query_pairs(rc, output_type="ndarray")
        d = x[p[:, 1]] - x[p[:, 0]]
        d -= np.rint(d / L) * L
        r2 = (d.astype(q) ** 2).sum(1)
        use = r2 <= min(rc * rc, 2.0 ** (1 / 3) if potential == "wca" else np.inf)
        d, r2 = d[use], r2[use]
        s6 = 1 / r2 ** 3
        e, w = 4 * (s6 * s6 - s6) - shift, 24 * (2 * s6 * s6 - s6)
        i2 = 1.0 / (d * d).sum(1)
        t6 = i2 * i2 * i2
        own = [np.asarray(4.0 * (t6 * t6 - t6) - float(shift) - e, dtype=np.float64),
               np.asarray(24.0 * (2.0 * t6 * t6 - t6) - w, dtype=np.float64)]
        with gpulib.MidpointLJ(L, [len(x)], precision="fp64", rc=rc, potential=potential) as s:
            s.set_atoms(x)
            _, ep, vir = s.forces(energy=True)
        exact = [e.sum(), w.sum()]
        rel.append([float((q(v[0]) - z) / abs(z)) for v, z in zip((ep, vir), exact)])
        allow = max(allow, *(np.sqrt(len(d)) * o.std() / abs(float(z)) for o, z in zip(own, exact)))
    rms = np.sqrt(np.mean(np.square(rel), axis=0))
    # (1 u: the last sums' 0.41 u with room for eight samples; lj_shifted: its shift is a double, whose own rounding
    # is in every pair)
    tol = U + 2 * allow + (U * len(d) * abs(float(shift)) / abs(float(exact[0])) if potential == "lj_shifted" else 0.0)
    assert (rms <= tol).all(), (rms / U, tol / U)


@pytest.mark.parametrize("sigma,rc", [(0.42, 0.32), (0.04, 0.1)])
def test_short_cutoff_in_large_cells(gpulib, oracle, sigma, rc):
    """A type pair whose cutoff is a sixtieth of the cell edge or less, in tiles of 14 cells: pairs just inside it, on
    both sides of the face where the tile's FP32 coordinates are largest, are the oracle's, each of them."""
    rng = np.random.default_rng(8)
    cross = 0.5 * (1.0 + sigma)
    lj = dict(ntypes=2, eps=[[1.0, cross], [cross, sigma]], sigma=[[1.0, cross], [cross, sigma]],
              rc=[[2.5, 2.5 * cross], [2.5 * cross, rc]])
    n, nbox = 250, 24
    boxes, parts = [], []
    for _ in range(nbox):
        L = 14 * 19.9 + rng.uniform(0.0, 4.0, 3)
        c = np.stack([np.zeros(n), rng.permutation(n) * (L[1] / n), (np.arange(n) + 0.5) * (L[2] / n)], 1)
        u = np.stack([np.ones(n), rng.uniform(-0.02, 0.02, n), rng.uniform(-0.02, 0.02, n)], 1)
        u /= np.sqrt((u * u).sum(1))[:, None]
        r = rc * (1.0 - 10.0 ** rng.uniform(-9, -7, n))[:, None]
        s = rng.uniform(0.1, 0.9, n)[:, None]
        p = np.concatenate([c - s * r * u, c + (1 - s) * r * u]) % L
        parts.append(p)
        boxes.append(L)
    pos, boxes = np.concatenate(parts), np.array(boxes)
    with gpulib.MidpointLJ(boxes, [2 * n] * nbox, precision="fp64", block_length=19.9, tile=(14, 14, 14), **lj) as sysm:
        sysm.set_atoms(pos, np.ones(len(pos), dtype=np.int32))
        f = sysm.forces()[0]
        accepted = sysm.counters()["accepted"]
    want = 0
    for b in range(nbox):
        k = slice(2 * n * b, 2 * n * (b + 1))
        ref = oracle.forces_typed(pos[k], boxes[b], lj["rc"], types=np.ones(2 * n, dtype=np.int32), threads=0,
                                  block_length=19.900390625, **{x: lj[x] for x in ("eps", "sigma", "ntypes")})
        want += ref["counts"].accepted
        fr = ref["forces"]
        assert np.sqrt(((f[k] - fr) ** 2).sum(1)).max() <= TOL64 * np.sqrt((fr * fr).sum(1).mean())
    assert want > 0.98 * n * nbox and accepted == want


@pytest.mark.parametrize("tile", [2, 4])
@pytest.mark.parametrize("apart", [0.0, 0.5, 0.74])
def test_overlapping_atoms(gpulib, oracle, tile, apart):
    """Atoms at random, no nearer than `apart`: every tile, most or a few are the FP64 body's, in grids above and below
    its blocks.  Energies, counters and forces as the oracle's, each to the accuracy of its own atom's terms."""
    n = 12000
    L = np.full(3, (n / 0.6) ** (1.0 / 3.0))
    pos = gpulib.gen_random(n, L, apart, 13) if apart else np.random.default_rng(13).uniform(0.0, 1.0, (n, 3)) * L
    ref = oracle.forces_typed(pos, L, 2.5, threads=0)
    with gpulib.MidpointLJ(L, [n], precision="fp64", tile=(tile,) * 3) as s:
        s.set_atoms(pos)
        for _ in range(2):
            f, e, w = s.forces(energy=True)
        plain = s.forces()[0]
        cnt = s.counters()
    # an atom's largest term bounds its force's error: 60 terms' roundings and the separations', amplified 14 times;
    # a difference across the box's face is rounded at the box's scale, 2^-49, up to 14 times that over r
    from scipy.spatial import cKDTree
    p = cKDTree(pos, boxsize=L).query_pairs(2.5, output_type="ndarray")
    d = pos[p[:, 1]] - pos[p[:, 0]]
    d -= np.rint(d / L) * L
    r = np.sqrt((d * d).sum(1))
    t = 24.0 * (2.0 * r ** -13 + r ** -7) * (60 * 14 * 2.0 ** -53 + 14 * 2.0 ** -48 / r)
    size = np.zeros(n)
    np.add.at(size, p[:, 0], t)
    np.add.at(size, p[:, 1], t)
    for g in (f, plain):
        assert (np.abs(g - ref["forces"]).max(1) <= size).all()
    assert e[0] == pytest.approx(ref["epot"], rel=TOL64) and w[0] == pytest.approx(ref["virial"], rel=TOL64)
    assert cnt["candidates"] == ref["counts"].candidates and cnt["accepted"] == ref["counts"].accepted


@pytest.mark.parametrize("sigma", [500.0, 1.0, 1e-4])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_pruning_at_the_ends_of_fp16(gpulib, oracle, precision, sigma):
    """The enumeration prunes cells on FP16 gaps: lengths whose squares are beyond FP16's largest number and below its
    smallest, atoms on and next to the cells' faces.  The same pairs as the oracle, which prunes nothing."""
    rng = np.random.default_rng(4)
    L = np.array([11.3, 12.5, 13.7]) * sigma
    h = 1.25 * sigma
    unit = 2.0 ** (np.floor(np.log2(h)) - 13)
    edge = float(np.ceil(h / unit) * unit)
    pos = gpulib.gen_random(1200, L / sigma, 0.85, 6) * sigma
    k = rng.integers(0, 1200, 500)
    a = rng.integers(0, 3, 500)
    pos[k, a] = np.floor(pos[k, a] / edge) * edge + rng.choice([0.0, 1e-9, -1e-9, 1e-6, -1e-6], 500) * sigma
    pos %= L
    from scipy.spatial import cKDTree
    close = cKDTree(pos, boxsize=L).query_pairs(0.8 * sigma, output_type="ndarray")
    keep = np.ones(len(pos), dtype=bool)
    keep[close[:, 1]] = False
    pos = np.ascontiguousarray(pos[keep])
    lj = dict(eps=sigma, sigma=sigma)  # forces of about 1
    ref = oracle.forces_typed(pos, L, 2.5 * sigma, threads=0, block_length=edge, **lj)
    with gpulib.MidpointLJ(L, [len(pos)], precision=precision, rc=2.5 * sigma, **lj) as s:
        s.set_atoms(pos)
        f = s.forces()[0]
        cnt = s.counters()
    assert cnt["candidates"] == ref["counts"].candidates and cnt["accepted"] == ref["counts"].accepted
    d, fr = np.sqrt(((f - ref["forces"]) ** 2).sum(1)), np.sqrt((ref["forces"] ** 2).sum(1).mean())
    assert d.max() <= TOL64 * fr if precision == "fp64" else np.sqrt((d * d).mean()) <= 1e-5 * fr
