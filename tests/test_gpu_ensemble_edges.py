"""GPU tests of the ensemble's kernels at their edges: direct sums of 1 to 1024
bodies (64 per block, sources in pairs, slices of the sources) at every block
size, energies of systems around the 1024-body chunk, boxes that grow for
several bodies, and two ensembles of different direct sizes alive together."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = 0.02


@pytest.fixture(scope="module")
def hc():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from nemo_gb300 import build as B
    B.build()
    from nemo_gb300 import hackcode
    return hackcode


def _systems(counts, seed, spread=1.0):
    rng = np.random.default_rng(seed)
    m = [rng.uniform(0.5, 1.5, k) / k for k in counts]
    ph = [rng.normal(0.0, spread, (k, 2, 3)) for k in counts]
    return m, ph


def _direct(m, x):
    d = x[None] - x[:, None]
    r2 = (d * d).sum(2) + EPS * EPS
    w = m[None] / np.sqrt(r2)
    np.fill_diagonal(w, 0.0)
    return ((w / r2)[:, :, None] * d).sum(1), -w.sum(1)


COUNTS = [1, 2, 3, 31, 33, 63, 64, 65, 127, 129, 1023, 1024]


@pytest.mark.parametrize("threads", [128, 256, 512])
def test_direct_sums_of_every_size(hc, threads):
    m, ph = _systems(COUNTS, 1)
    big = hc.Ensemble([2, 3000], eps=EPS, direct_max=4096)       # needs more shared memory than the next
    ens = hc.Ensemble(COUNTS, eps=EPS, direct_max=1024)
    ens.set_tuning(direct_threads=threads)
    ens.upload(np.concatenate(m), np.concatenate(ph))
    e = ens.step(1.0 / 64, 0, energy=True)
    _, acc, phi = ens.download(phase=False)
    off = np.concatenate([[0], np.cumsum(COUNTS)])
    for s, k in enumerate(COUNTS):
        a, p = _direct(m[s], ph[s][:, 0])
        ga, gp = acc[off[s]:off[s + 1]], phi[off[s]:off[s + 1]]
        # FP32 terms, hi + lo separations, compensated sums: the repository's 1e-5 per body
        assert (np.linalg.norm(ga - a, axis=1) <= 1e-5 * np.linalg.norm(a, axis=1)).all(), k
        assert (np.abs(gp - p) <= 1e-5 * np.abs(p)).all(), k
        ke = 0.5 * np.sum(m[s] * (ph[s][:, 1] ** 2).sum(1))
        np.testing.assert_allclose(e[s], [ke, 0.5 * np.sum(m[s] * gp), ke + 0.5 * np.sum(m[s] * gp)], rtol=1e-12)
    mb, pb = _systems([2, 3000], 2)
    big.upload(np.concatenate(mb), np.concatenate(pb))
    big.step(1.0 / 64, 0)
    _, acc, _ = big.download(phase=False, phi=False)
    a, _ = _direct(mb[1], pb[1][:, 0])
    assert (np.linalg.norm(acc[2:] - a, axis=1) <= 1e-5 * np.linalg.norm(a, axis=1)).all()
    big.close()
    ens.close()


def test_boxes_energies_and_caller_order(hc):
    """Tree systems around the kernels' chunks, with bodies far outside the first box (several rounds of the
    replay, in chunks before and after the first 2048): each as the single-system path has it."""
    counts = [1100, 40, 2047, 2049, 4097]
    m, ph = _systems(counts, 3)
    for s in (0, 2, 4):
        ph[s][5, 0] = (3.0, -2.5, 1.0)
        ph[s][counts[s] - 1, 0] = (-11.0, 4.0, 30.0)
    ens = hc.Ensemble(counts, tol=0.6, eps=EPS, direct_max=64)
    ens.upload(np.concatenate(m), np.concatenate(ph))
    e = ens.step(1.0 / 64, 0, energy=True)
    _, acc, phi = ens.download(phase=False)
    off = np.concatenate([[0], np.cumsum(counts)])
    for s, k in enumerate(counts):
        ga, gp = acc[off[s]:off[s + 1]], phi[off[s]:off[s + 1]]
        if k > 64:
            with hc.Context(k, tol=0.6, eps=EPS) as ctx:
                ctx.set_grouping("tree")
                ctx.upload(m[s], ph[s])
                ctx.evaluate()
                _, a, p = ctx.download(phase=False)
        else:
            a, p = _direct(m[s], ph[s][:, 0])
        rel = np.linalg.norm(ga - a, axis=1) / np.linalg.norm(a, axis=1)
        assert np.quantile(rel, 0.999) < 1e-5 and rel.max() < 1e-3, k
        ke = 0.5 * np.sum(m[s] * (ph[s][:, 1] ** 2).sum(1))
        np.testing.assert_allclose(e[s][:2], [ke, 0.5 * np.sum(m[s] * gp)], rtol=1e-12)
    ens.close()
