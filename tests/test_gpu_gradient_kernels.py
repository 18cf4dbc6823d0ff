"""The gradient kernels with two chains per lane, on as many observations as
they are chosen for (the last quad of observations partial): four warps up to
256 points and where blocks of 512 would be half empty, eight warps at 300 and
2,048, and at 33 parameters, whose sums leave room for one block on an SM."""
import numpy as np
import pytest

from gpumetropolis_b200 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,p,n_obs", [("logistic", 16, 300001), ("logistic", 16, 300002),
                                          ("poisson", 24, 200003), ("logistic", 31, 200001)])
def test_two_chains_per_lane(gpu, name, p, n_obs):
    w = W.make(name, n_obs=n_obs, p=p)
    m = w.model
    d = m.n_params
    rng = np.random.default_rng(n_obs)
    pts = w.truth["beta"] + rng.normal(0, 0.05, (2048, d))
    keep = np.array([0, 1, 31, 32, 63, 64, 128, 255, 256, 299, 511, 512, 599, 2047])
    og, oa = O.grad_abs_batch(m.loglik.code, m.loglik.consts, d, w.data, m.n_cols, n_obs,
                              pts[keep])
    same = []
    with gpu.Session(m.loglik.code, m.loglik.consts, m.prior.code, m.prior.consts, d, w.data,
                     m.n_cols, n_obs) as s:
        for n in (33, 64, 65, 128, 129, 256, 300, 600, 2048):
            g = s.grad_batch(pts[:n]).reshape(n, d)
            k = keep < n
            assert np.max(np.abs(g[keep[k]] - og[k]) / oa[k]) <= 1e-5, n
            if n > 128:  # one warp per chain: the same FP32 blocks whatever the kernel
                same.append(g[keep[:7]])
    # sums in FP64 of up to a few thousand partials, divided otherwise
    for g in same[1:]:
        assert np.max(np.abs(g - same[0]) / oa[:7]) <= 1e-12
