"""GPU tests of the team walk (several warps per group in systems with few
groups).  Massless bodies far away add targets but neither cells nor massive
groups, so the same massive bodies are walked by teams without them and by one
warp per group with them: the same decisions and counts, and forces that differ
by the order of their FP32 sums."""
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


def _run(hc, m, pos, criterion, theta, quad, grouping, prev):
    n = len(m)
    ph = np.zeros((n, 2, 3))
    ph[:, 0] = pos
    with hc.Context(n, tol=0.6, eps=0.02, usequad=quad, count_per_body=True) as ctx:
        ctx.upload(m, ph)
        ctx.set_box((-8.0, -8.0, -8.0), 16.0)
        ctx.set_grouping(grouping)
        if criterion != "body":
            ctx.set_criterion(criterion, theta)
        ctx.set_forces(prev)
        ctx.evaluate()
        _, acc, phi = ctx.download(phase=False)
        return acc, phi, ctx.body_counts()


# groups around the rule's lines: 1 group, 152 (16 warps), 380 (8), 1824 (4), more (1)
@pytest.mark.parametrize("n", [5, 200, 4864, 4865, 12161, 33000, 58369])
@pytest.mark.parametrize("criterion,theta,quad,grouping",
                         [("body", 0.0, True, "consecutive"), ("body", 0.0, False, "tree"), ("group", 0.6, True, "tree"),
                          ("error", 0.05, False, "tree"), ("error", 0.05, True, "tree"), ("barnes", 0.8, True, "tree")])
def test_team_walk_is_the_group_walk(hc, n, criterion, theta, quad, grouping):
    rng = np.random.default_rng(n)
    pos = rng.normal(0.0, 0.5, (n, 3)) * rng.uniform(0.1, 2.0, (n, 1))
    m = rng.uniform(0.5, 1.5, n) / n
    prev = -pos / (np.linalg.norm(pos, axis=1)[:, None] + 0.3) ** 3
    a, p, (b, c) = _run(hc, m, pos, criterion, theta, quad, grouping, prev)
    extra = 80000
    far = rng.uniform(6.0, 7.9, (extra, 3))
    a1, p1, (b1, c1) = _run(hc, np.concatenate([m, np.zeros(extra)]), np.concatenate([pos, far]), criterion, theta, quad,
                            grouping, np.concatenate([prev, np.full((extra, 3), 0.1)]))
    assert np.array_equal(b, b1[:n]) and np.array_equal(c, c1[:n])
    # FP32 partial sums of 64 terms, compensated: 64 * 2^-24 of the sum of magnitudes; accelerations cancel, so
    # their scale is the potential's
    scale = np.abs(p1[:n])
    assert (np.abs(p - p1[:n]) <= 4e-6 * scale).all()
    size = np.linalg.norm(a1[:n], axis=1) + scale
    assert (np.linalg.norm(a - a1[:n], axis=1) <= 4e-6 * size / 0.02).all()
    assert np.median(np.linalg.norm(a - a1[:n], axis=1) / np.linalg.norm(a1[:n], axis=1)) <= 1e-6


# so many massless bodies that the second run is one warp per group whatever the
# grouping: more than 16 table groups (12 of consecutive bodies) per SM
@pytest.mark.parametrize("n", [5, 200, 513, 4865, 12161])
@pytest.mark.parametrize("criterion,theta,quad,grouping",
                         [("body", 0.0, True, "consecutive"), ("body", 0.0, False, "tree"), ("group", 0.6, True, "tree"),
                          ("error", 0.05, False, "tree"), ("error", 0.05, True, "tree"), ("barnes", 0.8, True, "tree")])
def test_team_walk_is_one_warps_walk(hc, n, criterion, theta, quad, grouping):
    import torch
    extra = 44 * 17 * torch.cuda.get_device_properties(0).multi_processor_count
    rng = np.random.default_rng([n, 1])
    pos = rng.normal(0.0, 0.5, (n, 3)) * rng.uniform(0.1, 2.0, (n, 1))
    m = rng.uniform(0.5, 1.5, n) / n
    prev = -pos / (np.linalg.norm(pos, axis=1)[:, None] + 0.3) ** 3
    a, p, (b, c) = _run(hc, m, pos, criterion, theta, quad, grouping, prev)
    far = rng.uniform(6.0, 7.9, (extra, 3))
    a1, p1, (b1, c1) = _run(hc, np.concatenate([m, np.zeros(extra)]), np.concatenate([pos, far]), criterion, theta, quad,
                            grouping, np.concatenate([prev, np.full((extra, 3), 0.1)]))
    assert np.array_equal(b, b1[:n]) and np.array_equal(c, c1[:n])
    # bounds as above: FP32 partial sums of 64 terms, compensated
    scale = np.abs(p1[:n])
    assert (np.abs(p - p1[:n]) <= 4e-6 * scale).all()
    size = np.linalg.norm(a1[:n], axis=1) + scale
    assert (np.linalg.norm(a - a1[:n], axis=1) <= 4e-6 * size / 0.02).all()
