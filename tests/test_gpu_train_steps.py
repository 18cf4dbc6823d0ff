"""Training runs whose steps are enqueued one by one and replayed from a graph:
the result depends on the steps and their rates only, whatever their split into
calls and stages; every width's tiles against the emulated gradients."""
import numpy as np
import pytest

from oracle import mlp_oracle as MO

pytestmark = pytest.mark.gpu


def _pairs(n, d, seed=0):
    rng = np.random.default_rng(seed)
    th = rng.normal(size=(n, d))
    return th, np.sin(th.sum(axis=1)) - 0.3 * (th ** 2).sum(axis=1)


@pytest.mark.parametrize("hidden,batch", [(128, 128), (256, 384), (512, 256)])
def test_split_of_a_schedule_does_not_matter(gpu, hidden, batch):
    th, ll = _pairs(700, 5)

    def fit(calls):
        net = gpu.Surrogate(5, hidden=hidden, batch=batch, seed=3)
        net.set_normalizer(np.zeros(5), np.ones(5), float(ll.mean()), float(ll.std()))
        loss = np.concatenate([net.train_stages(th, ll, st) for st in calls])
        p = net.params()
        net.close()
        return loss, p

    # 41 steps: twelve one by one, graphs of four, a last one by itself
    whole = fit([[(20, 3e-3), (0, 1.0), (14, 1e-3), (7, 1e-4)]])
    for calls in ([[(20, 3e-3)], [(14, 1e-3)], [(7, 1e-4)]],
                  [[(1, 3e-3)], [(19, 3e-3), (3, 1e-3)], [(11, 1e-3), (7, 1e-4)]]):
        got = fit(calls)
        assert np.array_equal(got[0], whole[0]) and np.array_equal(got[1], whole[1])
    assert whole[0][-5:].mean() < whole[0][:5].mean()


@pytest.mark.parametrize("d,hidden,batch,n", [(3, 128, 128, 77), (64, 128, 256, 256),
                                              (65, 256, 128, 128), (70, 512, 256, 200)])
def test_gradients_of_every_tile_shape(gpu, d, hidden, batch, n):
    th, ll = _pairs(n, d, seed=1)
    net = gpu.Surrogate(d, hidden=hidden, batch=batch, seed=2)
    net.set_normalizer(np.zeros(d), np.ones(d), 0.0, 1.0)
    p = net.params()
    g, loss = net.gradients(th, ll)
    net.close()
    ref_loss, ref = MO.forward_backward(p, d, hidden, MO.f32(th.astype(np.float32)),
                                        MO.f32(ll.astype(np.float32)))
    # both sides round the operands to BF16 at the same places; a sum in
    # another order can move a rounding (2^-9) of a few of an operand's values
    assert abs(loss - ref_loss) <= 1e-4 * abs(ref_loss)
    off = 0
    for r in ref:
        got = g[off:off + r.size].reshape(r.shape)
        off += r.size
        assert np.linalg.norm(got - r) <= 5e-3 * max(np.linalg.norm(r), 1e-30)
