"""GPU tests of the split walk: a walk group whose bounding box spreads over
the whole system opens every cell, exceeds its budget of iterations and is
walked in parts.

The system: a small dense core in one octant of the root box and five bodies in
each of the other seven.  The seven small cells are packed into one group of 35
bodies whose box covers the core, so with every group criterion its bodies
interact with all others directly: their accelerations are the direct sum's,
and their counts n - 1 body-body interactions.
"""
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


def _system(n, seed=5):
    rng = np.random.default_rng(seed)
    far = []
    for octant in range(7):                       # x most significant; octant 7 (+, +, +) holds the core
        sign = np.array([1 if octant & b else -1 for b in (4, 2, 1)])
        far.append(sign * rng.uniform(0.3, 1.9, (5, 3)))
    d = rng.normal(size=(n - 35, 3))
    r = 0.2 * rng.random(n - 35)
    core = 0.5 + d / np.linalg.norm(d, axis=1)[:, None] * r[:, None]
    pos = np.concatenate([np.concatenate(far), core])
    order = rng.permutation(n)
    m = rng.uniform(0.5, 1.5, n) / n
    return m, pos[order], np.flatnonzero(order < 35)


def _direct(m, pos, idx, eps):
    acc, phi = np.zeros((len(idx), 3)), np.zeros(len(idx))
    for k, i in enumerate(idx):
        d = pos - pos[i]
        r2 = (d * d).sum(1) + eps * eps
        w = m / np.sqrt(r2)
        w[i] = 0.0
        acc[k], phi[k] = ((w / r2)[:, None] * d).sum(0), -w.sum()
    return acc, phi


# 4001: the smallest that exceeds the budget (35 bodies, 6000 nodes); 20011: few
# groups; 150001: as many groups as warps, tasks of several hundred bodies
@pytest.mark.parametrize("n", [4001, 20011, 150001])
@pytest.mark.parametrize("criterion,theta,quad", [("barnes", 0.8, False), ("group", 0.7, True), ("error", 0.05, True),
                                                  ("error", 0.05, False), ("learned", 0.05, True)])
def test_spread_group_is_the_direct_sum(hc, n, criterion, theta, quad):
    eps = 0.01
    m, pos, far = _system(n)
    phase = np.zeros((n, 2, 3))
    phase[:, 0] = pos
    got = []
    for graphs in (True, False):
        with hc.Context(n, tol=0.5, eps=eps, usequad=quad, count_per_body=True) as ctx:
            ctx.set_graphs(graphs)
            ctx.upload(m, phase)
            if criterion == "learned":
                ctx.learn_init(3)
            ctx.set_criterion(criterion, theta)
            for _ in range(3 if graphs else 2):  # accelerations of a previous evaluation from the second on
                ctx.evaluate()
                _, acc, phi = ctx.download(phase=False)
                got.append((acc, phi))
            b, c = ctx.body_counts()
            d = ctx.diagnostics()
        assert d.n2b == b.sum() and d.nbc == c.sum()
        assert (b[far] == n - 1).all() and (c[far] == 0).all()
    ea, ep = _direct(m, pos, far, eps)
    # FP32 sums of n terms, compensated every 64: the repository's 1e-5 per body
    assert (np.linalg.norm(acc[far] - ea, axis=1) <= 1e-5 * np.linalg.norm(ea, axis=1)).all()
    assert (np.abs(phi[far] - ep) <= 1e-5 * np.abs(ep)).all()
    # the same bits with and without graph replay, whatever warp ran what
    assert np.array_equal(got[1][0], got[4][0]) and np.array_equal(got[1][1], got[4][1])


def test_closing_kick_of_a_split_group(hc):
    """The combined parts end in the same closing half-kick as a whole walk's."""
    n, dt = 20011, 1.0 / 64
    m, pos, far = _system(n)
    phase = np.zeros((n, 2, 3))
    phase[:, 0] = pos
    with hc.Context(n, tol=0.5, eps=0.01) as ctx:
        ctx.upload(m, phase)
        ctx.set_criterion("barnes", 0.8)
        _, p0, a0, _ = ctx.step(dt, 0, snapshot=True)
        _, p1, a1, _ = ctx.step(dt, 1, snapshot=True)
    v_half = p0[:, 1] + 0.5 * dt * a0             # v1/2, then v1/2 + a0 dt/2 before the evaluation
    want = (v_half + 0.5 * dt * a0) + (a1 - a0) * (0.5 * dt)
    assert np.abs(p1[:, 1] - want)[far].max() <= 1e-13 * np.abs(want).max()


# prev: accelerations of a "previous evaluation", the same in both runs
@pytest.mark.parametrize("n,extra", [(4001, 2 ** 20), (20011, 3 * 2 ** 20)])
@pytest.mark.parametrize("criterion,theta", [("group", 0.7), ("error", 0.05), ("learned", 0.05)])
def test_statistics_count_a_given_up_walk_once(hc, n, extra, criterion, theta):
    """The spread group's walk is given up and walked in parts; the statistics are
    those of a walk in one piece.  That walk comes from the same bodies beside so
    many massless ones that the budget (it grows with the number of groups)
    holds; each of their groups of 64, far away, accepts the root: one candidate
    and one cell entry."""
    m, pos, _ = _system(n)
    prev = -pos / (np.linalg.norm(pos, axis=1)[:, None] + 0.3) ** 3
    rng = np.random.default_rng(2)
    got = []
    for k in (0, extra):
        phase = np.zeros((n + k, 2, 3))
        phase[:n, 0] = pos
        phase[n:, 0] = rng.uniform(1.0e4, 1.1e4, (k, 3))
        with hc.Context(n + k, tol=0.5, eps=0.01, usequad=True, count_per_body=True) as ctx:
            ctx.upload(np.concatenate([m, np.zeros(k)]), phase)
            ctx.set_forces(np.concatenate([prev, np.full((k, 3), 0.1)]))
            if criterion == "learned":
                ctx.learn_init(3)
            ctx.set_criterion(criterion, theta)
            ctx.evaluate()
            got.append(ctx.walk_stats())
    parts, whole = got
    groups = extra // 64
    hist = list(whole["mask_hist"])
    hist[32] -= groups
    assert parts["mask_hist"] == hist
    assert parts["candidates"] == whole["candidates"] - groups
    assert parts["entries_cell"] == whole["entries_cell"] - groups
    assert parts["entries_body"] == whole["entries_body"]
    assert parts["network"] == whole["network"] and (parts["network"] > 0) == (criterion == "learned")
