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
