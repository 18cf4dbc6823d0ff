"""Models whose linear predictor (six data columns and more) is an operand that
the paired code would fold into its consumer: a negation divided by a
parameter-only value, a product from which a softplus is taken.  They compile,
and the negations keep the tensor-core value kernel."""
import numpy as np
import pytest

from gpumetropolis_b200 import _native
from gpumetropolis_b200.build import build
from gpumetropolis_b200.dsl import gpum_model

P = 8
LIN = " + ".join(f"b{j} * x{j}" for j in range(1, P + 1))
NEGATED = {
    "gumbel": f"~ -(y - ({LIN})) / exp(s) - s - exp(-(y - ({LIN})) / exp(s))",
    "linear": f"~ -({LIN}) / exp(s) - s - log(1 + y^2)",
    "square": f"~ -(((-(y - ({LIN}))) / exp(s))^2) / 2 - s",
    "exponential": f"~ -exp(-({LIN}) / exp(s)) - y / exp(s) - s",
    "logistic": f"~ -log(1 + exp(-({LIN}) / s))",
    "mixture": f"~ log(0.3 * exp(-({LIN}) / s) + 0.7 * exp(-((y - s)^2) / 2))",
}
SCALED = {"scaled": f"~ 2 * ({LIN}) - log(1 + exp(s * y))"}


def _model(text):
    names = [f"{c}{j}" for c in "bx" for j in range(1, P + 1)]
    return gpum_model(text, params=names[:P] + ["s"], data=names[P:] + ["y"])


@pytest.mark.parametrize("name", sorted({**NEGATED, **SCALED}))
def test_folded_predictors_compile(name, tmp_path, monkeypatch):
    build()
    monkeypatch.setenv("GPUM_B200_CACHE", str(tmp_path))
    m = _model({**NEGATED, **SCALED}[name])
    assert _native.compile_check(m.loglik.code, m.loglik.consts, m.prior.code, m.prior.consts,
                                 m.n_params, m.n_cols) > 0


@pytest.mark.gpu
@pytest.mark.parametrize("n_obs,n_points", [(257, 3), (3001, 130)])
@pytest.mark.parametrize("name", sorted({**NEGATED, **SCALED}))
def test_folded_predictors_match_the_oracle(gpu, name, n_obs, n_points):
    from oracle import oracle as O
    m = _model({**NEGATED, **SCALED}[name])
    rng = np.random.default_rng(n_obs)
    beta = rng.normal(0, 0.3, P)
    data = rng.normal(0, 1, (n_obs, P + 1))
    data[:, P] += data[:, :P] @ beta
    data = data.astype(np.float32).astype(np.float64)
    pts = np.append(beta, 0.75) + rng.normal(0, 0.05, (n_points, P + 1))
    pts = pts.astype(np.float32).astype(np.float64)
    args = (m.loglik.code, m.loglik.consts, m.n_params, data, m.n_cols, n_obs, pts)
    with gpu.Session(m.loglik.code, m.loglik.consts, m.prior.code, m.prior.consts, m.n_params,
                     data, m.n_cols, n_obs, engine=1) as s:
        assert s.engine == 1
        if name in NEGATED:
            assert s.tensor_cores
        val, grad = s.loglik_batch(pts), s.grad_batch(pts).reshape(n_points, -1)
    # a dozen f32 roundings (2^-24 each) a term, of intermediates whose size is
    # at most 4 |l_i| + 4
    size = (4 * np.abs(O.loglik_pointwise(*args)).reshape(n_points, n_obs) + 4).sum(axis=1)
    assert np.max(np.abs(val - O.loglik_batch(*args)) / size) <= 12 * 2.0 ** -24
    og, oa = O.grad_abs_batch(*args)
    assert np.max(np.abs(grad - og) / np.maximum(oa, 1e-30)) <= 1e-5
