"""GPU tests of the octree build at the sizes and mixtures where its kernels
change form: the one-block sort's capacities, tile edges of the sort, the box
test, the compaction and the node emission, systems with massless bodies (the
compaction pass) and with many ties of the 63-bit high keys.  The tree is the
oracle's bit for bit, and a walk on tree groups made after the build gives the
same counts as one made with it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def hc():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from nemo_gb300 import build as B
    B.build()
    from nemo_gb300 import hackcode
    return hackcode


@pytest.fixture(scope="module")
def O():
    from oracle import oracle
    oracle.build(ref=None)
    return oracle


def _bodies(n, kind, seed):
    rng = np.random.default_rng([seed, n])
    pos = rng.normal(0.0, 0.7, (n, 3))
    m = rng.uniform(0.5, 1.5, n) / n
    if kind == "massless":
        m[rng.random(n) < 0.3] = 0.0
        if n > 3:
            m[:2] = 0.0                          # the first massive body is not the first body
    elif kind == "ties":                         # pairs and triples far closer than the high keys resolve
        k = n // 3
        pos[k:2 * k] = pos[:k] + rng.normal(0.0, 1e-6, (k, 3))
        pos[2 * k:3 * k] = pos[:k] + rng.normal(0.0, 1e-6, (k, 3))
    elif kind == "far":                          # many bodies outside the first box
        pos *= rng.uniform(0.1, 9.0, (n, 1)) ** 2
    return m, pos


def _canon(d):
    k = np.lexsort((d["corner"][:, 2], d["corner"][:, 1], d["corner"][:, 0], d["level"]))
    return {f: d[f][k] for f in ("level", "corner", "count", "mass", "cm")}


# sort: 1024, 2048, 4096, 8192 per form, 4096 per tile; box 4096, compaction and emission 2048 per tile
SIZES = [1, 2, 3, 31, 33, 1023, 1024, 1025, 2049, 4096, 4097, 8191, 8192, 8193, 20481]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("kind", ["plain", "massless", "ties", "far"])
def test_tree_matches_oracle(hc, O, n, kind):
    m, pos = _bodies(n, kind, 3)
    ph = np.zeros((n, 2, 3))
    ph[:, 0] = pos
    T = O.Tree(n, 12.0)
    assert T.build(m, pos, True) == 0
    ref = T.dump()
    with hc.Context(n, tol=0.6, eps=0.02, fcells=12.0, usequad=True, count_per_body=True) as ctx:
        ctx.upload(m, ph)
        ctx.build_tree()
        rmin, rsize = ctx.box()
        assert np.array_equal(rmin, T.box()[0]) and rsize == T.box()[1]
        c, r = _canon(ctx.dump_tree()), _canon(ref)
        for f in c:
            assert np.array_equal(c[f], r[f]), f
        assert ctx.tree_info().nbody_massive == int((m != 0).sum())
        _, _, rb, rc = T.forces(0.6, 0.02, True)
        ctx.forces()
        b, cc = ctx.body_counts()
        assert np.array_equal(b, rb) and np.array_equal(cc, rc)
        ctx.set_grouping("tree")                 # the table is made by the walk: the build had no use for it
        ctx.forces()
        b, cc = ctx.body_counts()
        assert np.array_equal(b, rb) and np.array_equal(cc, rc)
        ctx.evaluate()                           # made with the build
        b, cc = ctx.body_counts()
        assert np.array_equal(b, rb) and np.array_equal(cc, rc)


@pytest.mark.parametrize("n", [1, 31, 1024, 1025, 8192, 8193])
def test_points_of_any_number(hc, O, n):
    """Forces at n test points (the sort's forms without ties) equal the oracle's."""
    m, pos = _bodies(500, "plain", 4)
    pts = np.random.default_rng(n).normal(0.0, 1.5, (n, 3))
    ph = np.zeros((500, 2, 3))
    ph[:, 0] = pos
    T = O.Tree(500, 2.0)
    assert T.build(m, pos, True) == 0
    ra, rp = T.forces(0.6, 0.02, True, test_pos=pts, skip_self=False)[:2]
    with hc.Context(500, tol=0.6, eps=0.02, usequad=True) as ctx:
        ctx.upload(m, ph)
        ctx.build_tree()
        a, p = ctx.forces_at(pts)
    assert (np.linalg.norm(a - ra, axis=1) <= 1e-5 * np.linalg.norm(ra, axis=1)).mean() >= 0.999
    assert (np.abs(p - rp) <= 1e-5 * np.abs(rp)).mean() >= 0.999


# the passes' tiles: 1024 keys to 2^15 bodies, 2048 to 2^18, then 4096
@pytest.mark.parametrize("n", [9216, 9217, 32768, 32769, 34817, 262144, 262145])
@pytest.mark.parametrize("kind", ["massless", "ties"])
def test_tree_at_the_passes_tile_sizes(hc, O, n, kind):
    m, pos = _bodies(n, kind, 5)
    ph = np.zeros((n, 2, 3))
    ph[:, 0] = pos
    T = O.Tree(n, 12.0)
    assert T.build(m, pos, True) == 0
    ref = T.dump()
    with hc.Context(n, tol=0.6, eps=0.02, fcells=12.0, usequad=True) as ctx:
        ctx.upload(m, ph)
        ctx.build_tree()
        c, r = _canon(ctx.dump_tree()), _canon(ref)
        for f in c:
            assert np.array_equal(c[f], r[f]), f


def test_test_points_fewer_than_before_in_one_context(hc):
    """A context that served more test points serves fewer of them as a fresh one
    does: below 2^18 and 2^15 points the sort's tiles are smaller and more."""
    n = 3000
    m, ph = hc.mkplummer(n, 4)
    test = np.random.default_rng(6).uniform(-1.5, 1.5, (300000, 3))

    def fresh():
        ctx = hc.Context(n, tol=0.7, eps=0.05, usequad=True)
        ctx.upload(m, ph)
        ctx.build_tree()
        return ctx

    with fresh() as one:
        for k in (40000, 30000, 300000, 200000, 262144, 32768):
            acc, phi = one.forces_at(test[:k])
            with fresh() as ctx:
                a, p = ctx.forces_at(test[:k])
            assert np.array_equal(acc, a) and np.array_equal(phi, p), k


def _chain_bodies(n, far):
    """One body near the origin, the second at `far` on every axis (the box of
    size 4 at (-2, -2, -2) doubles until it reaches it), the others between."""
    rng = np.random.default_rng([n, int(far)])
    pos = far * rng.uniform(0.1, 1.0, (n, 3))
    pos[0], pos[1] = (0.1, -0.2, 0.3), far
    return rng.uniform(0.5, 1.5, n) / n, pos


# a box of 4 * 2^k: one-body cells down to level k - 1, the body one deeper
@pytest.mark.parametrize("n", [2, 5, 20000])
@pytest.mark.parametrize("k", [30, 31, 32])
def test_expansion_chain_to_the_last_level(hc, O, n, k):
    m, pos = _chain_bodies(n, 0.7 * 4.0 * 2.0 ** k)
    ph = np.zeros((n, 2, 3))
    ph[:, 0] = pos
    T = O.Tree(n, 40.0)
    assert T.build(m, pos, False) == 0
    ref = _canon(T.dump())
    assert ref["level"].max() == k - 1
    ra, rp, rb, rc = T.forces(0.6, 0.02, False)
    with hc.Context(n, tol=0.6, eps=0.02, fcells=40.0, usequad=False, count_per_body=True) as ctx:
        ctx.upload(m, ph)
        for _ in range(2):                       # captured, then replayed
            ctx.set_box((-2.0, -2.0, -2.0), 4.0)
            ctx.evaluate()
        assert ctx.box()[1] == T.box()[1]
        got = _canon(ctx.dump_tree())
        for f in got:
            if f != "quad":
                assert np.array_equal(got[f], ref[f]), f
        b, c = ctx.body_counts()
        _, a, p = ctx.download(phase=False)
    assert np.array_equal(b, rb) and np.array_equal(c, rc)
    assert (np.linalg.norm(a - ra, axis=1) <= 1e-5 * np.linalg.norm(ra, axis=1)).all()
    assert (np.abs(p - rp) <= 1e-5 * np.abs(rp)).all()


@pytest.mark.parametrize("n", [5, 20000])
@pytest.mark.parametrize("k", [33, 36, 60])
def test_expansion_chain_below_the_last_level_is_refused(hc, n, k):
    m, pos = _chain_bodies(n, 0.7 * 4.0 * 2.0 ** k)
    ph = np.zeros((n, 2, 3))
    ph[:, 0] = pos
    with hc.Context(n, tol=0.6, eps=0.02, fcells=40.0) as ctx:
        ctx.upload(m, ph)
        for call in (ctx.build_tree, ctx.evaluate, ctx.evaluate):
            with pytest.raises(hc.HCError) as e:
                call()
            assert e.value.code == -1 and "level %d" % (k - 1) in str(e.value)
            assert ctx.box()[1] == 4.0           # as it was
        ctx.set_box((-2.0, -2.0, -2.0), 4.0 * 2.0 ** k)      # held from the start: no chain
        ctx.evaluate()
        assert ctx.tree_info().max_level <= 30


@pytest.mark.parametrize("n", [200, 5000, 60000])
@pytest.mark.parametrize("criterion", ["group", "error"])
def test_body_rule_on_a_tree_built_for_larger_groups(hc, O, n, criterion):
    """The group criteria's table holds groups of up to 64 bodies, the per-body
    rule walks at most 32 together: on a tree built for the one, the other's walk
    over tree groups visits every body, and the group walk afterwards is the same
    as before it."""
    m, pos = _bodies(n, "plain", 7)
    ph = np.zeros((n, 2, 3))
    ph[:, 0] = pos
    T = O.Tree(n, 12.0)
    assert T.build(m, pos, True) == 0
    ra, rp, rb, rc = T.forces(0.6, 0.02, True)
    with hc.Context(n, tol=0.6, eps=0.02, fcells=12.0, usequad=True, count_per_body=True) as ctx:
        ctx.upload(m, ph)
        ctx.set_criterion(criterion, 0.5)
        ctx.build_tree()
        ctx.forces()
        first = ctx.download(phase=False)[1:] + ctx.body_counts()
        ctx.set_criterion("body", 0.0)
        ctx.set_grouping("tree")
        ctx.forces()
        _, a, p = ctx.download(phase=False)
        b, c = ctx.body_counts()
        assert np.array_equal(b, rb) and np.array_equal(c, rc)
        assert (np.linalg.norm(a - ra, axis=1) <= 1e-5 * np.linalg.norm(ra, axis=1)).mean() >= 0.999
        assert (np.abs(p - rp) <= 1e-5 * np.abs(rp)).all()
        ctx.set_criterion(criterion, 0.5)
        ctx.set_forces(np.zeros((n, 3)))          # as before the first walk: the error rule reads them
        ctx.forces()
        again = ctx.download(phase=False)[1:] + ctx.body_counts()
        for x, y in zip(first, again):
            assert np.array_equal(x, y)


@pytest.mark.parametrize("n", [300, 8192, 8193, 40000])
def test_long_runs_of_equal_high_keys(hc, O, n):
    """Runs of 2 to 60 bodies (and, massless, of a hundred outside the box) that only
    the low keys tell apart, in every order."""
    rng = np.random.default_rng(n)
    m, pos = _bodies(n, "plain", 8)
    pos = np.clip(pos, -1.9, 1.9)                # the box stays the first one, of size 4
    at = 0
    for k in (2, 3, 7, 31, 60):
        # within one cell of 2^-21 of the box: its corner from the first body
        cell = 4.0 / (1 << 21)
        box = np.floor((pos[at] + 64.0) / cell) * cell - 64.0
        pos[at:at + k] = box + cell * rng.choice(512, (k, 1), replace=False) / 512.0 * np.ones(3)
        at += k
    m[at:at + 100], pos[at:at + 100] = 0.0, 60.0 + rng.random((100, 3))
    ph = np.zeros((n, 2, 3))
    ph[:, 0] = pos
    T = O.Tree(n, 60.0)
    assert T.build(m, pos, True) == 0
    with hc.Context(n, tol=0.6, eps=0.02, fcells=60.0, usequad=True) as ctx:
        ctx.upload(m, ph)
        ctx.build_tree()
        c, r = _canon(ctx.dump_tree()), _canon(T.dump())
        for f in ("level", "corner", "count", "mass", "cm"):
            assert np.array_equal(c[f], r[f]), f
