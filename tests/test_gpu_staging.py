"""Results that reach the host through the pinned blocks (staging.hpp): at the
edges of a block (2^18 floats), with more chunks than blocks, and the same
draws into pageable and pinned memory; runs of one session whose sizes, kind
and length change, which keep or rebuild the captured graph."""
import threading

import numpy as np
import pytest

from gpumetropolis_b200 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu
BLOCK = 1 << 18


def _session(gpu, w):
    m = w.model
    return gpu.Session(m.loglik.code, m.loglik.consts, m.prior.code, m.prior.consts, m.n_params,
                       w.data, m.n_cols, w.n_obs)


@pytest.mark.parametrize("n_obs,n_points", [(1, 1), (2047, 2), (BLOCK - 1, 1), (BLOCK, 1),
                                            (BLOCK + 1, 1), (BLOCK // 2 + 3, 5),
                                            (BLOCK - 1, 19)])
def test_pointwise_blocks(gpu, n_obs, n_points):
    w = W.make("gaussian", n_obs=n_obs)
    m = w.model
    pts = np.linspace(3.0, 4.0, n_points).reshape(-1, 1)
    with _session(gpu, w) as s:
        got = s.loglik_pointwise(pts).reshape(n_points, n_obs)
        one = np.stack([s.loglik_pointwise(pts[k:k + 1]) for k in (0, n_points - 1)])
    # one value per observation, whatever the other points: equal bits
    assert np.array_equal(got[[0, n_points - 1]], one)
    ref = O.loglik_pointwise(m.loglik.code, m.loglik.consts, 1, w.data, 1, n_obs, pts)
    # three f32 roundings of values and of a difference below 16
    assert np.max(np.abs(got.ravel() - ref)) <= 1e-5 * max(1.0, np.max(np.abs(ref)))


@pytest.mark.parametrize("n_obs", [BLOCK // 2 - 1, BLOCK // 2, BLOCK // 2 + 1, 4 * BLOCK - 1,
                                   4 * BLOCK, 4 * BLOCK + 1])
def test_pointwise_pieces(gpu, n_obs):
    """Half-block pieces below four blocks, whole blocks and threads from there."""
    w = W.make("gaussian", n_obs=n_obs)
    m = w.model
    pts = np.array([[3.25]])
    with _session(gpu, w) as s:
        got = s.loglik_pointwise(pts)
    ref = O.loglik_pointwise(m.loglik.code, m.loglik.consts, 1, w.data, 1, n_obs, pts)
    assert np.max(np.abs(got - ref)) <= 1e-5 * max(1.0, np.max(np.abs(ref)))


def test_pointwise_from_two_threads(gpu):
    w = W.make("gaussian", n_obs=BLOCK + 5)
    pts = np.linspace(3.0, 4.0, 12).reshape(-1, 1)
    out = {}

    def go(k):
        with _session(gpu, w) as s:
            out[k] = [s.loglik_pointwise(pts) for _ in range(3)]

    ts = [threading.Thread(target=go, args=(k,)) for k in range(2)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    for k in range(2):
        for v in out[k]:
            assert np.array_equal(v, out[0][0])


@pytest.mark.parametrize("C,n_iter", [(1, 5), (300, 40), (4096, 70)])
def test_draws_to_pinned_and_pageable(gpu, C, n_iter):
    torch = pytest.importorskip("torch")
    w = W.make("logistic", n_obs=500, p=3)
    d = w.model.n_params
    init = w.truth["beta"] + 0.01 * np.random.default_rng(1).standard_normal((C, d))
    args = (init, np.full((C, d), 0.05), np.ones(C), n_iter, 3, 0)
    buf = torch.empty(C * d * n_iter, dtype=torch.float32, pin_memory=True).numpy()
    with _session(gpu, w) as s:
        a, acc, last = s.run(*args)
        b, acc2, last2 = s.run(*args, out_draws=buf)
    assert np.array_equal(a, b) and np.array_equal(acc, acc2) and np.array_equal(last, last2)


def test_one_session_many_runs(gpu):
    """Runs that reuse the captured graph and runs that cannot give what a
    session of their own gives."""
    w = W.make("logistic", n_obs=700, p=3)
    d = w.model.n_params
    rng = np.random.default_rng(2)
    runs = []
    for C, n_iter, seed, mode, rate in [(8, 40, 1, 0, 0.05), (8, 40, 2, 0, 0.1), (8, 90, 3, 0, 0.1),
                                        (8, 40, 4, 2, 0.1), (8, 40, 5, 3, 0.1), (9, 33, 6, 3, 0.1),
                                        (8, 40, 7, 1, 0.1), (8, 40, 8, 0, 0.1), (700, 40, 9, 0, 0.1),
                                        (8, 31, 10, 0, 0.1), (8, 64, 11, 0, 0.1)]:
        init = w.truth["beta"] + 0.05 * rng.standard_normal((C, d))
        L = np.tile(0.1 * np.eye(d), (C, 1, 1)) if mode in (2, 3) else None
        runs.append((init, np.full((C, d), rate), np.ones(C), n_iter, seed, mode, 0.4, 1e-3, L))
    with _session(gpu, w) as s:
        shared = []
        for r in runs:
            shared.append(s.run(*r))
            s.loglik_batch(r[0][:3])  # evaluation buffers used in between
    for r, got in zip(runs, shared):
        with _session(gpu, w) as s:
            alone = s.run(*r)
        for x, y in zip(got, alone):
            assert np.array_equal(x, y)
