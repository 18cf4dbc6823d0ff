"""Narrow models: several tiles per shared-memory stage (eight of 256
observations for one column), and the exact folds of the paired code."""
import numpy as np
import pytest

from gpumetropolis_b200 import workloads as W
from gpumetropolis_b200.dsl import gpum_model
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("engine", [2, 0])
@pytest.mark.parametrize("n_obs,n_points", [(1, 3), (255, 3), (257, 40), (2048, 5), (2049, 5),
                                            (4097, 300), (300001, 512), (1000003, 2)])
def test_sums_across_stage_edges(gpu, n_obs, n_points, engine):
    w = W.make("gaussian", n_obs=n_obs)
    m = w.model
    pts = np.linspace(2.5, 4.5, n_points).reshape(-1, 1)
    keep = np.unique(np.linspace(0, n_points - 1, 5).astype(int))
    with gpu.Session(m.loglik.code, m.loglik.consts, m.prior.code, m.prior.consts, 1, w.data, 1,
                     n_obs, engine=engine) as s:
        got = s.loglik_batch(pts)
    ref = O.loglik_batch(m.loglik.code, m.loglik.consts, 1, w.data, 1, n_obs, pts[keep])
    # every term is <= 0, so the sum's relative error is that of its terms:
    # the f32 rounding of y and mu against a difference of a few units
    assert np.max(np.abs(got[keep] - ref)) <= 1e-6 * np.max(np.abs(ref)) + 1e-5


def test_log_sum_of_two_underflows(gpu):
    w = W.make("mixture", n_obs=64)
    m = w.model
    y = np.array([1e30, -1e30, np.inf, np.nan, 0.0, -2.0, 1e-30, 3.0])
    pts = np.array([[0.3, -2.0, 3.0, 0.1, 0.4]])
    args = (m.loglik.code, m.loglik.consts, m.n_params, y.reshape(-1, 1), 1, y.size)
    with gpu.Session(m.loglik.code, m.loglik.consts, m.prior.code, m.prior.consts, m.n_params,
                     y.reshape(-1, 1), 1, y.size, engine=1) as s:
        got = s.loglik_pointwise(pts)
    # (y - mu)^2 overflows FP32: both terms are -inf, and so is their sum
    assert np.all(np.isneginf(got[:3])) and np.isnan(got[3])
    ref = O.loglik_pointwise(*args, pts)
    np.testing.assert_allclose(got[4:], ref[4:], rtol=2e-6)


@pytest.mark.parametrize("text", [
    "~ -2.5 * log(1 + ((y - b) / exp(s))^2 / 4)",
    "~ -2.5 * log(((y - b) / exp(s))^2 / 8 + 3)",
    "~ -((y - b)^2) / exp(s) - b - log(0.5 + y^2 / 1024)",
    "~ b - y / 4 - -(y * b) / s",
])
def test_folds_match_the_oracle(gpu, text):
    rng = np.random.default_rng(5)
    y = np.concatenate([rng.normal(0, 3, 900), [0.0, 1e-22, -1e-22, 1e10, -1e10, 1e-40]])
    y = y.astype(np.float32).astype(np.float64)
    m = gpum_model(text, params=["b", "s"], data="y")
    pts = np.array([[0.25, 0.5], [0.0, 1.0], [-1.5, 0.125]])
    args = (m.loglik.code, m.loglik.consts, 2, y.reshape(-1, 1), 1, y.size)
    with gpu.Session(m.loglik.code, m.loglik.consts, m.prior.code, m.prior.consts, 2,
                     y.reshape(-1, 1), 1, y.size, engine=1) as s:
        got = s.loglik_pointwise(pts).reshape(3, -1)
        tot = s.loglik_batch(pts)
    ref = O.loglik_pointwise(*args, pts).reshape(3, -1)
    # a dozen f32 roundings (2^-24 each) of intermediates whose size is that of
    # the terms' absolute sum, here at most 4 |ref| + 4
    assert np.max(np.abs(got - ref) / (4 * np.abs(ref) + 4)) <= 12 * 2.0 ** -24
    assert np.max(np.abs(tot - got.sum(axis=1)) / np.abs(got).sum(axis=1)) <= 1e-6


@pytest.mark.parametrize("p,n_obs,n_points", [(3, 255, 70), (3, 513, 12), (3, 257, 9), (5, 64, 57),
                                              (40, 300, 70), (40, 300, 9)])
def test_interpreter_at_two_observations(gpu, p, n_obs, n_points):
    # eight chains at two observations per thread where the tile (256, or 128
    # and less for 41 columns) leaves every lane two, sixteen chains elsewhere
    w = W.make("logistic", n_obs=n_obs, p=p)
    m = w.model
    pts = w.truth["beta"] + np.random.default_rng(1).normal(0, 0.1, (n_points, m.n_params))
    args = (m.loglik.code, m.loglik.consts, m.n_params, w.data, m.n_cols, n_obs, pts)
    with gpu.Session(m.loglik.code, m.loglik.consts, m.prior.code, m.prior.consts, m.n_params,
                     w.data, m.n_cols, n_obs, engine=0) as s:
        got, tot = s.loglik_pointwise(pts), s.loglik_batch(pts)
    ref = O.loglik_pointwise(*args)
    # an f32 linear predictor of p + 1 terms of size below 4, two roundings each
    assert np.max(np.abs(got - ref)) <= 2 * (p + 8) * 4 * 2.0 ** -23
    ref = O.loglik_batch(*args)
    assert np.max(np.abs(tot - ref) / np.abs(ref)) <= 1e-6
