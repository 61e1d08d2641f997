"""Track blocks (csrc/tracks.cu): the choice of nodes and weights, restated in
numpy on synthetic formation tracks.

A block's nodes are picked by a Cholesky factorisation of the correlation
sinc(2 rho |u - u'|), pivoted on the worst predicted sample, until the mean
squared error of the weights -- interpolation and independent node errors of
2e-7 together -- is below 1.8 (2e-7)^2."""
import numpy as np
import pytest

from viss_optimize_3d_b200 import synth

NOISE = 2e-7          # relative error of a node value
EVALUATED = 3.7e-7    # of an exponential term of the direct kernels
T = 128


def nodes_and_weights(u, rho):
    n = len(u)
    G = np.sinc(2 * rho * np.linalg.norm(u[:, None] - u[None], axis=2))
    L, diag, used, piv, ld = np.zeros((n, n)), np.ones(n), np.zeros(n, bool), [], []
    while diag.max() > 4.5 * NOISE ** 2 or diag.mean() > 1.8 * NOISE ** 2:
        r = len(piv)
        if r == n * 3 // 4:
            return None, None
        p = int(np.argmax(np.where(used, -1.0, diag)))
        d = 1.0 - L[p, :r] @ L[p, :r]
        ld.append(np.sqrt(max(d, 0.0) + NOISE ** 2))
        L[:, r] = (G[:, p] - L[:, :r] @ L[p, :r]) / ld[-1]
        if r == 0 and np.all(G[:, p] == 1.0):           # one point: one node
            return [p], L[:, :1] / ld[-1]
        diag = np.maximum(diag - L[:, r] ** 2, 0.0)
        used[p] = True
        piv.append(p)
    r = len(piv)
    L11 = np.tril(L[piv, :r], -1) + np.diag(ld)
    return piv, np.linalg.solve(L11.T, L[:, :r].T).T


@pytest.mark.parametrize("name,pixels", [("c3_10mhz", 64), ("c3_10mhz", 128), ("c3_1mhz", 256), ("prod_1mhz", 1024)])
def test_predicted_samples_are_as_accurate_as_evaluated_ones(name, pixels):
    cfg = synth.CONFIGS[name]
    P = synth.satellite_positions(cfg)
    pairs = synth.baseline_pairs(cfg.n_sat)
    u_all = (P[:, pairs[:, 0]] - P[:, pairs[:, 1]]) / (synth.C_LIGHT / cfg.freqs_hz[0])
    side = np.sqrt(4 * np.pi / cfg.npix)
    nx = 2 ** int(np.ceil(np.log2(pixels) / 2))
    rng = np.random.default_rng(5)
    ranks, noise, bias = [], [], []
    for _ in range(6):
        b, t0 = rng.integers(len(pairs)), rng.integers(cfg.n_snap - T)
        u = u_all[t0:t0 + T, b]
        c = rng.standard_normal(3)
        c /= np.linalg.norm(c)
        e1 = np.cross(c, [0.3, -0.5, 0.8])
        e1 /= np.linalg.norm(e1)
        e2 = np.cross(c, e1)
        x, y = np.meshgrid((np.arange(nx) - (nx - 1) / 2) * side, (np.arange(pixels // nx) - (pixels / nx - 1) / 2) * side)
        s = c + x.reshape(-1, 1) * e1 + y.reshape(-1, 1) * e2
        d = s / np.linalg.norm(s, axis=1, keepdims=True) - c
        piv, W = nodes_and_weights(u, np.linalg.norm(d, axis=1).max())
        if piv is None:                 # the longest baselines on the larger groups: left to other sizes
            continue
        sky = np.exp(rng.standard_normal(pixels))
        V = np.exp(-2j * np.pi * (u @ d.T)) @ sky
        err = W @ V[piv] - V
        ranks.append(len(piv))
        bias.append(np.sqrt(np.mean(np.abs(err) ** 2) / np.sum(sky ** 2)))
        noise.append(np.mean(np.sum(W ** 2, axis=1)))
    assert len(ranks) >= 3
    # fewer nodes than samples, and a predicted sample (its weights' own error and
    # the nodes' together) no further off than an evaluated one
    assert max(ranks) <= T // 2 and np.mean(ranks) < 0.45 * T, ranks
    total = [np.hypot(e, NOISE * np.sqrt(n)) for e, n in zip(bias, noise)]
    assert max(total) < EVALUATED, (noise, bias)


def test_equal_samples_take_one_node():
    """Zero baselines: every sample is the same; one node whose FP32 weights are
    exactly one, so that sums of ones stay exact integers."""
    piv, W = nodes_and_weights(np.zeros((T, 3)), 0.05)
    assert len(piv) == 1
    assert np.all(W.astype(np.float32) == np.float32(1.0))
