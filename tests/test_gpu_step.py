"""The step kernel (partial sums, accept decision, draw, next proposal) against
the oracle sampler, at the chain counts where its warps per chain change, with
the Langevin factor staged in shared memory (24 parameters) and read from
global memory (120 parameters), and with more observation blocks than threads
of a chain's warps.
"""
import numpy as np
import pytest

from gpumetropolis_b200 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu

RWM, DE, CHOL, MALA = 0, 1, 2, 3


@pytest.mark.parametrize("p,n_obs,C,mode,engine", [
    (3, 70, 1, RWM, 2), (3, 70, 7, DE, 2), (3, 70, 592, CHOL, 2), (3, 70, 593, RWM, 2),
    (3, 70, 1185, MALA, 2), (3, 70, 2369, CHOL, 2), (3, 70, 4737, RWM, 2),
    (23, 70, 9, MALA, 2), (23, 70, 601, MALA, 0), (119, 70, 3, MALA, 2), (119, 70, 5, CHOL, 2),
    (3, 300001, 2, RWM, 2), (3, 300001, 2, MALA, 0),
    # the gradient kernel with two chains per lane: from 257 chains, up to 33
    # parameters (its last column of chains empty, half full, full)
    (23, 1027, 256, MALA, 2), (23, 1027, 257, MALA, 2), (23, 258, 512, MALA, 2),
    (32, 70, 545, MALA, 2), (33, 70, 545, MALA, 2),
])
def test_step_follows_the_oracle(gpu, p, n_obs, C, mode, engine):
    n_iter = 8 if n_obs < 1000 else 2 if n_obs > 2000 else 4
    w = W.make("logistic", n_obs=n_obs, p=p)
    m = w.model
    d = m.n_params
    rng = np.random.default_rng(C)
    scale = 1.0 / np.sqrt(n_obs * d)
    init = w.truth["beta"] + scale * rng.standard_normal((C, d))
    sd = np.full((C, d), scale)
    temps = np.linspace(1.0, 2.0, C)
    L = None
    if mode in (CHOL, MALA):
        L = scale * (np.eye(d) + 0.3 / np.sqrt(d) * np.tril(rng.standard_normal((C, d, d)), -1))
    args = (init, sd, temps, n_iter, 5, mode, 0.4, 1e-3, L)
    prog = (m.loglik.code, m.loglik.consts, m.prior.code, m.prior.consts, d, w.data, m.n_cols,
            w.n_obs)
    with gpu.Session(*prog, engine=engine) as s:
        g, acc, last = s.run(*args)
    o, _, _ = O.run(*prog, *args)
    g = g.reshape((n_iter, C, d), order="F")
    o = o.reshape((n_iter, C, d), order="F")
    # A decision can differ only where |log ratio - log u| is inside the error
    # of the two data sums, 1e-6 of sum |l_i| each (about 0.5 n_obs): at 70
    # observations below 1e-4 per step, 8e-4 per chain, at 1,027 below 1e-3 per
    # step at the bar and below 1e-4 at the 1e-7 that such sums have.  With 300,001 it is
    # 0.6 of a log unit at the bar (1e-8 of the sum in practice), so those
    # runs are two chains by two steps and compared as they are.
    same = np.all(np.isclose(g, o, rtol=1e-5, atol=1e-4 * scale * np.sqrt(d)), axis=(0, 2))
    assert np.sum(~same) <= int(4e-3 * C), np.nonzero(~same)
    lp = (O.loglik_batch(m.loglik.code, m.loglik.consts, d, w.data, m.n_cols, n_obs,
                         g[-1].astype(np.float64))
          + O.loglik_batch(m.prior.code, m.prior.consts, d, np.zeros(1), 1, 1,
                           g[-1].astype(np.float64)))
    # the state recorded in f32 moves the log posterior by its gradient times
    # 2^-24 |theta|, below 1e-6 n_obs; 1e-6 n_obs more for the FP32 sum
    assert np.max(np.abs(last - lp)) <= 2e-6 * n_obs
    assert 0.0 <= acc.min() and acc.max() <= 1.0


# The gradient kernel of four warps at the edges of its shared chains and of its
# range; values and gradient 3, 16 and 17 wide (sums of several observation
# blocks side by side up to 16).
@pytest.mark.parametrize("p,n_obs,n_points", [(1, 515, 32), (1, 2049, 33), (1, 300001, 64),
                                              (14, 515, 65), (14, 9001, 128), (14, 2049, 256),
                                              (15, 9001, 129), (15, 70, 257)])
def test_gradient_sums(gpu, p, n_obs, n_points):
    w = W.make("logistic", n_obs=n_obs, p=p)
    m = w.model
    pts = w.truth["beta"] + np.random.default_rng(4).normal(0, 0.1, (n_points, m.n_params))
    keep = np.unique(np.linspace(0, n_points - 1, 40).astype(int))
    prog = (m.loglik.code, m.loglik.consts, m.n_params, w.data, m.n_cols, w.n_obs)
    with gpu.Session(m.loglik.code, m.loglik.consts, m.prior.code, m.prior.consts, m.n_params,
                     w.data, m.n_cols, w.n_obs) as s:
        g = s.grad_batch(pts).reshape(n_points, -1)
    og, oa = O.grad_abs_batch(*prog, pts[keep])
    assert np.max(np.abs(g[keep] - og) / oa) <= 1e-5


# A partial quad is one warp's, however many share a chain: gradients with two
# chains per lane equal those with one bit for bit.
@pytest.mark.parametrize("n_obs", [1, 2, 3])
@pytest.mark.parametrize("n_points", [60, 300])
def test_partial_quad_of_two_chains(gpu, n_obs, n_points):
    w = W.make("logistic", n_obs=n_obs, p=16)
    m = w.model
    pts = np.random.default_rng(0).normal(0, 0.5, (n_points, m.n_params))
    with gpu.Session(m.loglik.code, m.loglik.consts, m.prior.code, m.prior.consts, m.n_params,
                     w.data, m.n_cols, w.n_obs) as s:
        two = s.grad_batch(pts).reshape(n_points, -1)
        one = np.concatenate([s.grad_batch(pts[k:k + 20]).reshape(20, -1)
                              for k in range(0, n_points, 20)])
    assert np.array_equal(two, one)


@pytest.mark.parametrize("n_obs,n_points", [(70, 1), (70, 593), (300001, 3), (9001, 4737)])
@pytest.mark.parametrize("engine", [2, 0])
def test_batch_sums(gpu, n_obs, n_points, engine):
    w = W.make("logistic", n_obs=n_obs, p=6)
    m = w.model
    rng = np.random.default_rng(3)
    pts = w.truth["beta"] + rng.normal(0, 0.1, (n_points, m.n_params))
    keep = np.unique(np.linspace(0, n_points - 1, 40).astype(int))
    prog = (m.loglik.code, m.loglik.consts, m.n_params, w.data, m.n_cols, w.n_obs)
    with gpu.Session(m.loglik.code, m.loglik.consts, m.prior.code, m.prior.consts, m.n_params,
                     w.data, m.n_cols, w.n_obs, engine=engine) as s:
        v, g = s.loglik_batch(pts), s.grad_batch(pts).reshape(n_points, -1)
    o = O.loglik_batch(*prog, pts[keep])
    og, oa = O.grad_abs_batch(*prog, pts[keep])
    assert np.max(np.abs(v[keep] - o) / np.abs(o)) <= 1e-6  # every term is below 0
    assert np.max(np.abs(g[keep] - og) / oa) <= 1e-5
