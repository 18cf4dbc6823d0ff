"""Sessions alive together whose launches of one kernel need different amounts
of shared memory: what one of them sets up leaves the other's calls as they
were."""
import threading

import numpy as np
import pytest

from gpumetropolis_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _session(gpu, w, engine=2):
    m = w.model
    return gpu.Session(m.loglik.code, m.loglik.consts, m.prior.code, m.prior.consts, m.n_params,
                       w.data, m.n_cols, w.n_obs, engine=engine)


@pytest.mark.parametrize("p", [16, 30])
def test_batches_of_two_sessions(gpu, p):
    w = W.make("logistic", n_obs=1031, p=p)
    pts = w.truth["beta"] + np.random.default_rng(0).normal(0, 0.1, (512, w.model.n_params))
    with _session(gpu, w, 0) as a, _session(gpu, w, 0) as b:
        first = a.loglik_batch(pts)
        small = b.loglik_batch(pts[:10])
        again = a.loglik_batch(pts)
    assert np.array_equal(first, again)
    assert np.allclose(small, first[:10], rtol=1e-6)  # FP32 terms, summed over other blocks


def _start(w, C, L_of):
    d = w.model.n_params
    init = w.truth["beta"] + 0.01 * np.random.default_rng(1).standard_normal((C, d))
    return (init, np.full((C, d), 0.01), np.ones(C), 6, 7, 2, 0.0, 0.0,
            np.tile(L_of * np.eye(d), (C, 1, 1)))


def test_prepared_runs_of_two_sessions(gpu):
    # Cholesky factors of 65 and of 55 parameters staged by the step kernel:
    # 72 and 52 KB a block
    wide, narrow = (W.make("logistic", n_obs=300, p=p) for p in (64, 54))
    C = 594
    ra, rb = _start(wide, C, 0.01), _start(narrow, C, 0.01)
    with _session(gpu, wide) as s:
        alone = s.run(*ra)
    with _session(gpu, wide) as a, _session(gpu, narrow) as b:
        a.prepare(*ra)
        b.prepare(*rb)
        a.advance(6)
        draws, acc, last, n = a.fetch()
        b.advance(6)
        assert b.fetch()[3] == 6
    assert n == 6
    assert np.array_equal(np.ravel(draws), np.ravel(alone[0]))
    assert np.array_equal(acc, alone[1]) and np.array_equal(last, alone[2])


def test_runs_beside_a_thread_that_opens_and_closes_sessions(gpu):
    # runs of 64 iterations capture a graph in each new session, training steps
    # in each call; the other thread allocates, grows and frees meanwhile
    w = W.make("logistic", n_obs=2000, p=5)
    d = w.model.n_params
    args = (np.tile(w.truth["beta"], (8, 1)), np.full((8, d), 0.05), np.ones(8), 64, 3, 0)
    pts = np.random.default_rng(0).normal(0, 1, (1000, d))
    stop, wrong, opened = threading.Event(), [], [0]

    def other():
        try:
            while not stop.is_set():
                with _session(gpu, w) as s:
                    for n in (4, 1000):
                        s.loglik_batch(pts[:n])
                    s.run(*args[:3], 5, 3, 0)
                opened[0] += 1
        except Exception as e:  # reported by the test below
            wrong.append(e)

    def once():
        net = gpu.Surrogate(d, hidden=128, batch=256, seed=1)
        with _session(gpu, w) as s:
            run = s.run(*args)
        net.train(pts, -np.sum(pts ** 2, axis=1), steps=40, lr=1e-3)
        params = net.params()
        net.close()
        return [*run, params]

    first = once()
    t = threading.Thread(target=other)
    t.start()
    try:
        runs = [once() for _ in range(30)]
    finally:
        stop.set()
        t.join()
    assert not wrong, wrong
    assert opened[0] > 0
    for r in runs:
        for x, y in zip(first, r):
            assert np.array_equal(x, y)
