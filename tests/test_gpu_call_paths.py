"""The routes of a force call, by size, kind of host array and grid.

- Calls at new positions of up to 16,384 atoms go through the context's own
  page-locked arrays as a replayed graph from the third call on.
- Page-locked arrays are read and written in place, also where their end is not
  a whole block of atoms and where they start off a 16-byte boundary; arrays off
  the doubles' own boundary are copied.
- Above 16,384 atoms the types are checked on the device.
- The FP64 form's default tiles are 4, 3 or 2 cells by the number of tiles, the
  mixed form's CTAs are wider where one wave holds the grid: the same pairs and
  forces as with the other choices.
"""
import numpy as np
import pytest

pytestmark = [pytest.mark.gpu]

TOL64 = 1e-12  # of F_rms, the FP64 form against the oracle
TOL_MIXED = 1e-5  # RMS


def frms(f):
    return np.sqrt((f * f).sum(1).mean())


def check(f, ref, precision):
    d = np.sqrt(((f - ref) ** 2).sum(1))
    if precision == "fp64":
        assert d.max() <= TOL64 * frms(ref)
    else:
        assert np.sqrt((d * d).mean()) <= TOL_MIXED * frms(ref)


def crystal(gpulib, n, seed=1):
    """n atoms of a jittered FCC box of at least that many."""
    m = 2
    while 4 * m ** 3 < n:
        m += 1
    pos, L = gpulib.gen_fcc(m, 0.8442)
    rng = np.random.default_rng(seed)
    return (pos[rng.permutation(len(pos))[:n]] + rng.uniform(-0.05, 0.05, (n, 3))) % L, np.full(3, L)


@pytest.mark.parametrize("n,precision,kw", [(2, "fp64", {}), (257, "fp64", {}), (257, "mixed", {}),
                                            (3000, "mixed", dict(pair_skin=0.3)), (16384, "mixed", {}),
                                            (16385, "fp64", {})])
def test_repeated_small_calls(gpulib, oracle, n, precision, kw):
    """New positions, new arrays and other results asked for at each call."""
    pos, L = crystal(gpulib, max(n, 256))
    pos = np.ascontiguousarray(pos[:n])
    if n == 2:
        pos[1] = (pos[0] + 0.7) % L
    rng = np.random.default_rng(5)
    with gpulib.MidpointLJ(L, [n], precision=precision, **kw) as s:
        s.set_atoms(pos)
        for call in range(9):
            p = (pos + rng.uniform(-0.02, 0.02, pos.shape)) % L
            ref = oracle.forces_typed(p, L, 2.5, threads=0)
            energy, acc = call % 2 == 1, call in (3, 6, 7)
            base = rng.uniform(-1, 1, pos.shape) if acc else np.zeros_like(pos)
            f, e, w = s.forces_at(p, out=base.copy(), accumulate=acc, energy=energy)
            check(f, base + ref["forces"], precision)
            if energy:
                tol = TOL64 if precision == "fp64" else 1e-6
                assert e[0] == pytest.approx(ref["epot"], rel=tol)
                # (the virial is a difference of two terms: of their size)
                assert abs(w[0] - ref["virial"]) <= tol * (abs(ref["virial"]) + 48 * abs(ref["epot"]))
            if call == 5:  # a run between the calls; the next positions follow on
                s.run(3, 0.001)


@pytest.mark.parametrize("n", [16385, 65537])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("shift", [0, 8, 4])
def test_arrays_in_place(gpulib, n, precision, shift):
    """Page-locked arrays `shift` bytes into their allocation against ordinary ones, bit for bit, with sentinels
    on both sides."""
    pos, L = crystal(gpulib, n)
    rng = np.random.default_rng(2)

    def page_locked(a):
        raw = gpulib.pinned_empty((a.size + 4,)).view(np.uint8)
        raw[:] = 0xAB
        v = raw[16 + shift:16 + shift + a.nbytes].view(np.float64).reshape(a.shape)
        v[...] = a
        return raw, v

    with gpulib.MidpointLJ(L, [n], precision=precision) as s:
        s.set_atoms(pos)
        for acc in (False, True, False):
            p = (pos + rng.uniform(-0.02, 0.02, pos.shape)) % L
            base = rng.uniform(-1, 1, pos.shape)
            want, _, _ = s.forces_at(p, out=base.copy(), accumulate=acc)
            here, _, _ = s.forces(out=base.copy(), accumulate=acc)
            assert np.array_equal(want, here)
            (praw, pv), (raw, f) = page_locked(p), page_locked(base)
            s.forces_at(pv, out=f, accumulate=acc)
            assert np.array_equal(f, want) and np.array_equal(pv, p)
            f[...] = base
            s.forces(out=f, accumulate=acc)
            assert np.array_equal(f, want)
            for r in (praw, raw):
                assert (r[:16 + shift] == 0xAB).all() and (r[16 + shift + p.nbytes:] == 0xAB).all()


@pytest.mark.parametrize("n", [16384, 16385])
def test_types_outside_the_table(gpulib, n):
    pos, L = crystal(gpulib, n)
    types = (np.arange(n) % 2).astype(np.int32)
    with gpulib.MidpointLJ(L, [n], ntypes=2) as s:
        s.set_atoms(pos, types)
        f, _, _ = s.forces()
        for bad, where in ((2, n - 1), (-1, 0)):
            t = types.copy()
            t[where] = bad
            with pytest.raises(gpulib.ExamdError):
                s.set_atoms(pos, t)
            s.set_atoms(pos, types)
            assert np.array_equal(s.forces()[0], f)


def test_batch_with_an_empty_box(gpulib, oracle):
    n = [9000, 0, 1, 8001]
    parts = [crystal(gpulib, max(k, 256), seed=k) for k in n]
    pos = np.concatenate([p[:k] for (p, _), k in zip(parts, n)])
    L = np.array([b for _, b in parts])
    types = (np.random.default_rng(3).random(len(pos)) < 0.4).astype(np.int32)
    lj = dict(ntypes=2, eps=[[1.0, 0.7], [0.7, 0.5]], sigma=[[1.0, 0.9], [0.9, 0.85]], rc=2.5)
    with gpulib.MidpointLJ(L, n, precision="fp64", **lj) as s:
        s.set_atoms(pos, types)
        f, e, _ = s.forces(energy=True)
    o = np.concatenate([[0], np.cumsum(n)])
    for b in (0, 3):
        k = slice(o[b], o[b + 1])
        ref = oracle.forces_typed(pos[k], L[b], types=types[k], threads=0, **lj)
        check(f[k], ref["forces"], "fp64")
        assert e[b] == pytest.approx(ref["epot"], rel=TOL64)
    assert not f[o[2]:o[3]].any() and e[1] == 0.0 and e[2] == 0.0


@pytest.mark.parametrize("m", [4, 10, 13, 20, 28])
def test_fp64_default_tiles(gpulib, m):
    """Boxes on both sides of the two lines of the default; tile 2 of the largest has more than one chunk of
    tile energies (4096)."""
    n = 4 * m ** 3
    pos, L = crystal(gpulib, n)
    out = []
    for kw in ({}, dict(tile=(4, 4, 4)), dict(tile=(2, 2, 2))):
        with gpulib.MidpointLJ(L, [n], precision="fp64", **kw) as s:
            s.set_atoms(pos)
            f, e, w = s.forces(energy=True)
            out.append((f, e[0], w[0], s.counters()))
    f, e, w, c = out[0]
    assert c["tiles"] in (out[1][3]["tiles"], out[2][3]["tiles"]) or out[1][3]["tiles"] < c["tiles"] < out[2][3]["tiles"]
    for g, eg, wg, cg in out[1:]:
        assert np.sqrt(((g - f) ** 2).sum(1)).max() <= TOL64 * frms(f)
        assert eg == pytest.approx(e, rel=TOL64) and abs(wg - w) <= TOL64 * (abs(w) + 48 * abs(e))
        assert cg["accepted"] == c["accepted"] and cg["candidates"] == c["candidates"]


@pytest.mark.parametrize("rc,tile", [(2.5, 4), (3.0, 3)])
def test_fp64_default_tiles_by_their_atoms(gpulib, rc, tile):
    """A box with tiles of 4 cells enough for the chip at either cutoff: at rc 3 they are too large for three CTAs."""
    n = 4 * 30 ** 3
    pos, L = crystal(gpulib, n)
    out = []
    for kw in ({}, dict(tile=(tile,) * 3), dict(tile=(7 - tile,) * 3)):
        with gpulib.MidpointLJ(L, [n], precision="fp64", rc=rc, **kw) as s:
            s.set_atoms(pos)
            out.append((s.forces()[0], s.counters()))
    assert out[0][1]["tiles"] == out[1][1]["tiles"] != out[2][1]["tiles"]
    for f, c in out[1:]:
        assert np.sqrt(((f - out[0][0]) ** 2).sum(1)).max() <= TOL64 * frms(out[0][0])
        assert c["accepted"] == out[0][1]["accepted"]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("m", [4, 14, 20, 24])
def test_warps_give_the_same_forces(gpulib, precision, m):
    """The default (wide CTAs, finer work units in few-wave grids) against 4 and 8 warps."""
    n = 4 * m ** 3
    pos, L = crystal(gpulib, n)
    out = []
    for kw in ({}, dict(warps=8), dict(warps=4)):
        with gpulib.MidpointLJ(L, [n], precision=precision, **kw) as s:
            s.set_atoms(pos)
            f, e, _ = s.forces(energy=True)
            plain, _, _ = s.forces()
            assert np.array_equal(f, plain)
            out.append((f, e[0]))
    for f, e in out[1:]:
        assert np.array_equal(f, out[0][0]) and e == pytest.approx(out[0][1], rel=TOL64)


@pytest.mark.parametrize("atoms", [2500, 2700, 3180, 3290])
def test_tiles_at_the_shared_memory_limit(gpulib, oracle, atoms):
    """FP64 tiles of 4 cells (6^3 of the box's 8^3 staged) of about this many atoms: with the passes' headroom (to
    2,617 atoms), without it, and beyond what the fixed-point pass's tables leave room for (3,216), where the FP64
    body takes every tile (to 3,336)."""
    rc, m = 5.0, 24
    L = np.full(3, 8 * rc / 2)
    g = (np.arange(m) + 0.5) * (L[0] / m)
    pos = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    rng = np.random.default_rng(atoms)
    n = int(atoms / (6 / 8) ** 3)
    pos = pos[rng.permutation(len(pos))[:n]] + rng.uniform(-0.02, 0.02, (n, 3))
    with gpulib.MidpointLJ(L, [n], precision="fp64", rc=rc, tile=(4, 4, 4)) as s:
        s.set_atoms(pos)
        f, e, _ = s.forces(energy=True)
        assert 0 <= s.counters()["max_tile_atoms"] - atoms <= 50
    ref = oracle.forces_typed(pos, L, rc, threads=0)
    check(f, ref["forces"], "fp64")
    assert e[0] == pytest.approx(ref["epot"], rel=TOL64)


def packed(gpulib, n, size, L, seed):
    """n atoms at random in a cube of `size` in the box's corner."""
    return np.ascontiguousarray(np.random.default_rng(seed).uniform(0.0, size, (n, 3)) % L)


@pytest.mark.parametrize("n,size", [(8000, 3.0), (3300, 3.7), (2900, 3.7)])
@pytest.mark.parametrize("before", [False, True])
def test_fixed_point_pass_after_a_crowded_tile(gpulib, n, size, before):
    """Atoms that no pass has room for in one tile (refused), or only the FP64 body; the next configuration is computed
    as by a context that never saw them, bit for bit (the fixed-point pass: FP64 sums would differ from run to run)."""
    L = np.full(3, 32.0)
    m = int(np.ceil(n ** (1 / 3)))
    g = (np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n] + 0.5) * (32.0 / m)
    good = g + np.random.default_rng(1).uniform(-0.1, 0.1, g.shape)
    bad = packed(gpulib, n, size, L, 2)
    with gpulib.MidpointLJ(L, [n], precision="fp64", tile=(3, 3, 3)) as s:
        s.set_atoms(good)
        want = [s.forces()[0], s.forces_at(good)[0], s.forces(energy=True)[0]]
        state = s.run(8, 0.001, graph_chunk=4) and s.state()
    with gpulib.MidpointLJ(L, [n], precision="fp64", tile=(3, 3, 3)) as s:
        if before:
            s.set_atoms(good)
            s.run(8, 0.001, graph_chunk=4)
        if n == 8000:
            for _ in range(2):
                with pytest.raises(gpulib.ExamdError):
                    s.set_atoms(bad)
        else:
            s.set_atoms(bad)
            s.forces()
        s.set_atoms(good)
        got = [s.forces()[0], s.forces_at(good)[0], s.forces(energy=True)[0]]
        for a, b in zip(got, want):
            assert np.array_equal(a, b)
        s.run(8, 0.001, graph_chunk=4)
        for a, b in zip(s.state(), state):
            assert np.array_equal(a, b)


def test_energies_of_many_boxes(gpulib):
    """An eager run with energies keeps a few MB of them (4 per array and three steps' more), however many boxes, and
    gives the energies of a run in graphs."""
    torch = pytest.importorskip("torch")
    n = 65535  # (the most whose energies are summed)
    rng = np.random.default_rng(1)
    with gpulib.MidpointLJ(np.full((n, 3), 6.25), np.ones(n, dtype=np.int64), precision="mixed") as s:
        pos, vel = rng.uniform(0.0, 6.25, (n, 3)), rng.normal(size=(n, 3))
        s.set_atoms(pos, vel=vel)
        s.run(2, 0.001)
        free = torch.cuda.mem_get_info()[0]
        a = s.run(7, 0.001, energies=True)
        # three arrays of 4 MB and three steps of 0.5 MB, each in 2 MB blocks
        assert free - torch.cuda.mem_get_info()[0] <= 3 * (4 + 3 * 0.53 + 2) * 2 ** 20
        s.set_atoms(pos, vel=vel)
        s.run(2, 0.001)
        b = s.run(7, 0.001, graph_chunk=2, energies=True)
    for k in ("ekin", "epot"):
        assert np.array_equal(a[k], b[k])
    assert np.allclose(a["ekin"], 0.5 * (vel ** 2).sum(1), rtol=1e-12) and not a["epot"].any()
