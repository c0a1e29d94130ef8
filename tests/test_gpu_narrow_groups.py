"""GPU tests of the group walk's second bodies.  A group of 33 to 64 bodies
gives every lane one body and lays its other 1 to 32 over 8, 16 or 32 lanes, the
free lanes taking other entries of the list; the walk that counts per body keeps
one entry for all lanes.  Both decide alike, so their forces differ by the order
of FP32 sums.  And of the softening's two forms of the inverse root."""
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


def _run(hc, m, pos, criterion, theta, quad, prev, count, eps=0.02):
    n = len(m)
    ph = np.zeros((n, 2, 3))
    ph[:, 0] = pos
    with hc.Context(n, tol=0.6, eps=eps, usequad=quad, count_per_body=count) as ctx:
        ctx.upload(m, ph)
        ctx.set_box((-8.0, -8.0, -8.0), 16.0)
        ctx.set_grouping("tree")
        if criterion != "body":
            ctx.set_criterion(criterion, theta)
        ctx.set_forces(prev)
        ctx.evaluate()
        _, acc, phi = ctx.download(phase=False)
        return acc, phi


# clusters of k bodies, one group each: teams of 16 and 4 warps, one warp a group
@pytest.mark.parametrize("clusters", [1, 60, 1000, 2600])
@pytest.mark.parametrize("k", [32, 33, 40, 41, 48, 49, 63, 64])
@pytest.mark.parametrize("criterion,theta,quad", [("group", 0.6, True), ("error", 0.05, True), ("barnes", 0.8, True), ("group", 0.6, False)])
def test_second_bodies_narrow_and_wide(hc, clusters, k, criterion, theta, quad):
    rng = np.random.default_rng(100 * clusters + k)
    side = 16                                                   # cells of size 1, a cluster in the middle of each
    at = rng.choice(side ** 3, clusters, replace=False)
    centre = np.stack([at // side ** 2, at // side % side, at % side], 1) - 7.5
    pos = (centre[:, None] + rng.uniform(-0.3, 0.3, (clusters, k, 3))).reshape(-1, 3)
    m = rng.uniform(0.5, 1.5, len(pos)) / len(pos)
    prev = -pos / (np.linalg.norm(pos, axis=1)[:, None] + 0.3) ** 3
    a, p = _run(hc, m, pos, criterion, theta, quad, prev, False)
    a1, p1 = _run(hc, m, pos, criterion, theta, quad, prev, True)
    # FP32 partial sums of 64 terms, compensated: 64 * 2^-24 of the sum of magnitudes; accelerations cancel, so
    # their scale is the potential's
    scale = np.abs(p1)
    assert (np.abs(p - p1) <= 4e-6 * scale).all()
    size = np.linalg.norm(a1, axis=1) + scale
    assert (np.linalg.norm(a - a1, axis=1) <= 4e-6 * size / 0.02).all()
    assert np.median(np.linalg.norm(a - a1, axis=1) / np.linalg.norm(a1, axis=1)) <= 1e-6


@pytest.mark.parametrize("criterion,theta", [("body", 0.0), ("group", 0.6), ("error", 0.05)])
@pytest.mark.parametrize("quad", [False, True])
def test_softenings_on_both_sides_of_the_smallest_normal_square(hc, criterion, theta, quad):
    """1e-19 squared is a denormal FP32 number and 1.1e-19 squared is not: the
    lists take their inverse roots by different instructions.  Neither changes a
    separation of these bodies (1e-19 against 1e-7 and more), so nor any bit."""
    rng = np.random.default_rng(3)
    pos = rng.normal(0.0, 1.0, (20000, 3)).clip(-7.5, 7.5)
    m = rng.uniform(0.5, 1.5, len(pos)) / len(pos)
    prev = -pos / (np.linalg.norm(pos, axis=1)[:, None] + 0.3) ** 3
    a, p = _run(hc, m, pos, criterion, theta, quad, prev, False, eps=1.0e-19)
    a1, p1 = _run(hc, m, pos, criterion, theta, quad, prev, False, eps=1.1e-19)
    assert np.isfinite(p).all() and np.array_equal(p, p1) and np.array_equal(a, a1)
