"""The walk at the sizes where its batches and lane layouts change: targets of
1 .. 65 particles (odd and even, one to 32 lane groups, past the largest walk
group), source batches with remainders, both expansions, with and without the
r^2 = 0 mask.  Interaction counts equal the oracle's; forces within the
suite's bounds (FP64 1e-12, split 1e-5 of the global norm)."""
import numpy as np
import pytest

import bhg
from helpers import cube, rel_error
from oracle import Params, soa
from test_gpu_parity import _oracle_build

pytestmark = pytest.mark.gpu

SIZES = [2, 3, 31, 32, 33, 63, 64, 65, 127, 129, 191, 193, 257, 1021, 4099]


@pytest.mark.parametrize("precision,tol", [(bhg.PRECISION_FP64, 1e-12), (bhg.PRECISION_SPLIT, 1e-5)])
@pytest.mark.parametrize("leaf", [1, 2, 3, 5, 7, 16, 31, 33, 64, 65, 300])
def test_walk_sizes_match_oracle(gpu, oracle, leaf, precision, tol):
    for n in SIZES:
        parts = cube(n, 100 + n, spread=3.0)
        dom, sk, perm, mp, t = _oracle_build(oracle, parts, leaf)
        tg = oracle.targets(t, leaf, 1024)
        for quad, eps2 in ((True, 1e-4), (True, 0.0), (False, 1e-4), (False, 0.0)):
            racc, counts = oracle.walk(t, tg, soa(mp), [Params(0.6, eps2, 1.0, int(quad))] * len(tg))
            gpu.upload(parts)
            gpu.stats(reset=True)
            gpu.build_tree(leaf, 1024)
            gpu.compute_multipoles()
            acc = gpu.walk_forces(bhg.Context.params(0.6, eps2, 1.0, quad, precision), leaf)
            st = gpu.stats()
            assert (st["pp"], st["pc"]) == (int(counts[0]), int(counts[1])), (n, quad, eps2)
            assert np.all(np.isfinite(acc))
            assert rel_error(acc, racc) <= tol, (n, quad, eps2)


@pytest.mark.parametrize("precision,tol", [(bhg.PRECISION_FP64, 1e-12), (bhg.PRECISION_SPLIT, 1e-5)])
def test_leaf_too_large_for_a_list_entry(gpu, oracle, precision, tol):
    """300 particles at one point: a leaf of more particles than a partial
    list's entry counts, which some targets of the groups around it open."""
    parts = cube(2000, 41)
    parts["pos"][:300] = [1.25, -3.5, 2.0]
    dom, sk, perm, mp, t = _oracle_build(oracle, parts, 8)
    tg = oracle.targets(t, 8, 1024)
    for theta in (0.3, 0.6):
        racc, counts = oracle.walk(t, tg, soa(mp), [Params(theta, 1e-4, 1.0, 1)] * len(tg))
        gpu.upload(parts)
        gpu.stats(reset=True)
        gpu.build_tree(8, 1024)
        gpu.compute_multipoles()
        acc = gpu.walk_forces(bhg.Context.params(theta, 1e-4, 1.0, True, precision), 8)
        st = gpu.stats()
        assert (st["pp"], st["pc"]) == (int(counts[0]), int(counts[1]))
        assert rel_error(acc, racc) <= tol


@pytest.mark.parametrize("precision", [bhg.PRECISION_SPLIT, bhg.PRECISION_FP64])
def test_full_lists_give_the_same_bits_in_both_schedules(precision):
    """theta 0.15 with one particle per leaf fills both lists of most groups,
    so their traversals pause and go on; the two-pass schedule (all slots) and
    the one-pass schedule (a budget with few slots) agree bit for bit."""
    parts = cube(20000, 5)
    fp = bhg.Context.params(0.15, 1e-6, 1.0, True, precision)
    out = []
    for budget in (0, 36 << 20):
        with bhg.Context(device=0, hbm_budget=budget) as ctx:
            ctx.upload(parts)
            ctx.step(fp, 1, 64, 1, 0.01, 0.01)
            out.append(ctx.download().tobytes())
    assert out[0] == out[1]


@pytest.mark.parametrize("precision", [bhg.PRECISION_SPLIT, bhg.PRECISION_FP64])
@pytest.mark.parametrize("n,leaf,theta,budget", [(30000, 16, 0.2, 25), (65536, 16, 0.3, 40), (60000, 32, 0.25, 36)])
def test_paused_traversals_beside_dense_jobs(n, leaf, theta, budget, precision):
    """Few groups whose dense lists fill up, at leaf sizes with fewer node records
    than particles: the group's own job evaluates its lists and goes on in
    another one while its dense job may still read the first.  The same counts
    and bits as the one-pass schedule without dense jobs (a budget of few lists)."""
    parts = bhg.plummer(n, 600 + leaf)[0]
    fp = bhg.Context.params(theta, 1e-4, 1.0, True, precision)
    out = []
    for mb in (0, budget):
        with bhg.Context(device=0, hbm_budget=mb << 20) as ctx:
            ctx.upload(parts)
            ctx.step(fp, leaf, 256, leaf, 0.01, 0.01)
            s = ctx.stats()
            out.append((ctx.download().tobytes(), s["pp"], s["pc"]))
    assert out[0] == out[1]


@pytest.mark.parametrize("ns", [1, 2, 3, 127, 129, 256, 257, 700])
def test_direct_sum_rows_and_splits(gpu, oracle, ns):
    """Row counts around the block's (1 .. 256 rows, a remainder block), source
    counts below a tile, with remainders and over many splits, of the second
    of two systems, softened and not."""
    for n in (701, 1024, 1283, 50021):
        a, b = cube(300, 3), cube(n, 4, spread=2.0)
        idx = np.sort(np.random.default_rng(ns).choice(n, ns, replace=False)).astype(np.uint32)
        gpu.upload_systems([a, b])
        for eps2 in (1e-4, 0.0):
            assert rel_error(gpu.direct_sum(idx, eps2, G=0.5, system=1), oracle.direct(soa(b), idx, eps2, 0.5)) < 1e-13


def test_repeated_shapes_give_the_same_bits():
    """A shape's first evaluation runs kernel by kernel, its second is captured
    and later ones replay the graph, across uploads, other shapes in between
    (same particle count, other systems) and systems leaving (the state moves
    to the other buffer): the same bits every time."""
    one, two = cube(3000, 61), [cube(1300, 62), cube(1700, 63)]
    fp = bhg.Context.params(0.5, 1e-4)
    ref = {}
    with bhg.Context(device=0) as ctx:
        for what in "aaaabbbbabaabbrrrr":
            if what == "a":
                ctx.upload(one)
            else:
                ctx.upload_systems(two)
            if what == "r":
                ctx.remove_systems([ctx.system_ids()[0]])
            for _ in range(2 if what == "r" else 1):
                ctx.step(fp, 8, 256, 16, 0.01, 0.02)
            got = ctx.download().tobytes()
            assert ref.setdefault(what, got) == got, what


@pytest.mark.parametrize("leaf", [1, 2, 16, 255, 5000])
def test_topology_sizes_match_oracle(gpu, oracle, leaf):
    """The octree at particle counts around a warp's, a unit's and a tile's
    share, with runs of equal keys (depth-21 leaves) across them."""
    for n in (1, 2, 31, 33, 255, 257, 511, 513, 4095, 4097, 8193):
        parts = cube(n, 200 + n)
        parts["pos"][n // 3: n // 3 + n // 5] = parts["pos"][0]
        dom, sk, perm, mp, t = _oracle_build(oracle, parts, leaf)
        gpu.upload(parts)
        gpu.build_tree(leaf, 256)
        gpu.compute_multipoles()
        g = gpu.tree()
        assert g["n"] == t["n"], n
        for k in ("begin", "count", "first_child", "nchild", "leaf", "depth"):
            assert np.array_equal(g[k], t[k][:t["n"]]), (n, k)
        for k in ("center", "hw", "mass", "com", "iab"):
            assert np.array_equal(g[k], np.asarray(t[k][:t["n"]]), equal_nan=True), (n, k)


@pytest.mark.parametrize("n", [1, 127, 128, 129, 3000, 65541])
def test_snapshot_sizes_match_oracle(oracle, n):
    """Snapshots around a tile's particles, in one part and in several, into a
    buffer that holds any snapshot (copied as it is formatted) and into one of
    exactly its size; one byte less is refused."""
    parts = cube(n, 70 + n, spread=1e-3)
    parts["vel"] = np.random.default_rng(n).normal(size=(n, 3)) * 10.0 ** np.random.default_rng(n).integers(-9, 9, (n, 1))
    want = oracle.write_vtk(parts)
    with bhg.Context(device=0) as ctx:
        ctx.upload(parts)
        assert ctx.snapshot_vtk() == want
        exact = np.zeros(len(want), np.uint8)
        assert ctx.snapshot_vtk_into(exact) == len(want) and exact.tobytes() == want
        with pytest.raises(bhg.BhgError):
            ctx.snapshot_vtk_into(np.zeros(len(want) - 1, np.uint8))


@pytest.mark.parametrize("precision", [bhg.PRECISION_SPLIT, bhg.PRECISION_FP64])
def test_softening_of_others_changes_no_bits(precision):
    """Softened and unsoftened systems in one context: each as it is alone, with
    few walk groups and with many."""
    for sizes in ((3000, 700, 1500, 1), (60000, 30000, 200000)):
        systems = [cube(n, 80 + i, spread=2.0) for i, n in enumerate(sizes)]
        eps2 = [1e-4 if i % 2 == 0 else 0.0 for i in range(len(sizes))]
        fp = bhg.Context.params(0.5, 0.0, 1.0, True, precision)

        def run(ctx, which):
            ctx.upload_systems([systems[i] for i in which])
            k = len(which)
            ctx.set_system_params([0.6] * k, [eps2[i] for i in which], [0.01] * k, [0.02] * k)
            ctx.stats()
            for _ in range(2):
                ctx.step_systems(fp, 16, 256, 16)
            s = ctx.stats()
            return np.split(ctx.download(), np.cumsum([sizes[i] for i in which])[:-1]), s["pp"], s["pc"]

        with bhg.Context(device=0) as ctx:
            mixed, pp, pc = run(ctx, range(len(sizes)))
            alone = [run(ctx, [i]) for i in range(len(sizes))]
        assert (pp, pc) == (sum(a[1] for a in alone), sum(a[2] for a in alone))
        for i, a in enumerate(alone):
            assert mixed[i].tobytes() == a[0][0].tobytes(), i


@pytest.mark.parametrize("n", [2, 3, 5, 8, 10])
def test_sources_of_one_record_add_in_64_bits(n):
    """Up to ten particles in one leaf: a lane evaluates one record of two
    sources for a target, so no two FP32 terms share a partial sum, and the
    forces of all sources together are those of each alone (the others
    massless) added in FP64: n additions of 2^-53 each, not 2^-24."""
    parts = cube(n, 500 + n)
    parts["mass"] = np.random.default_rng(n).uniform(0.5, 2.0, n)
    fp = bhg.Context.params(0.5, 1e-4)

    with bhg.Context(device=0) as ctx:
        def forces(mass):
            p = parts.copy()
            p["mass"] = mass
            ctx.upload(p)
            ctx.build_tree(16, 256)
            ctx.compute_multipoles()
            return ctx.walk_forces(fp, 16)

        alone = np.array([forces(np.where(np.arange(n) == i, parts["mass"], 0.0)) for i in range(n)])
        together = forces(parts["mass"])
    assert np.all(np.abs(together - alone.sum(0)) <= 2 * n * 2.0**-53 * np.abs(alone).sum(0))
