"""Two-stage runs on both sides of the one-block screen (up to 2,048 chains):
a random-walk chain's stream and proposals depend on the seed and its number
only, so the first chains of a larger run are those of a smaller one."""
import numpy as np
import pytest

from gpumetropolis_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fitted(gpu):
    w = W.make("logistic", n_obs=3001, p=4)
    m = w.model
    s = gpu.Session(m.loglik.code, m.loglik.consts, m.prior.code, m.prior.consts, m.n_params,
                    w.data, m.n_cols, w.n_obs)
    rng = np.random.default_rng(4)
    C, d = 2050, m.n_params
    init = w.truth["beta"] + 0.04 * rng.standard_normal((C, d))
    s.record(40000)
    s.run(init, np.full((C, d), 0.05), np.ones(C), 20, 1, 0)
    net = gpu.Surrogate(d, hidden=128, batch=1024, seed=1)
    s.train_surrogate(net, [(150, 3e-3), (100, 1e-3)])
    s.record(0)
    yield s, net, init
    net.close()
    s.close()


def _run(fitted, C, mode=0):
    s, net, init = fitted
    d = init.shape[1]
    sd = np.full((C, d), 0.08)
    L = np.tile(0.08 * np.eye(d), (C, 1, 1)) if mode == 2 else None
    n = 20
    draws, acc, last, exact = s.run_da(net, init[:C], sd, np.ones(C), n, 9, mode, proposal_l=L)
    return draws.reshape((n, C, d), order="F"), acc, last, exact


@pytest.mark.parametrize("C", [1, 31, 33, 1024, 1025, 2047, 2048])
def test_screen_equals_the_separate_kernels(fitted, C):
    big = _run(fitted, 2050)  # three kernels
    got = _run(fitted, C)     # one
    assert 0 < big[3].sum() < 20 * 2050  # some screened out, some not
    assert np.array_equal(got[3], big[3][:C])
    assert np.array_equal(got[0], big[0][:, :C])
    assert np.array_equal(got[1], big[1][:C])
    # partial sums are split over other blocks: f64 rounding only
    assert np.max(np.abs(got[2] - big[2][:C])) <= 1e-9 * np.max(np.abs(big[2]))


def test_cholesky_with_the_identity_is_the_diagonal_walk(fitted):
    a, b = _run(fitted, 500, 0), _run(fitted, 500, 2)
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[3], b[3])
