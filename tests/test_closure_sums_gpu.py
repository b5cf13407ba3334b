"""The closure's gradient, loss and training kernels at the edges of their
blocks: one sample, ragged last blocks, odd counts, more blocks than CTAs are
resident (a CTA then runs several).

Tolerances: the gradient's operands are rounded to TF32 (2^-11 each) in at
most four chained products, 8 * 2^-11 in all; the loss is an FP32 forward
pass per sample, 1e-5. A training iteration is compared with Adam in FP64 on
the library's own gradient of the same minibatch: its FP32 operations move a
parameter of magnitude below 4 by at most one unit in the last place (2.4e-7)
beside 1e-5 of the step.
"""
import numpy as np
import pytest

from test_closure_gpu import _features, _split

pytestmark = pytest.mark.gpu


def _targets(x, seed):
    xs = x / x.std(0)
    return np.abs(3e-4 * np.log1p(np.exp(0.8 * xs[:, 0] - 0.6 * xs[:, 6])) + np.random.default_rng(seed).normal(0, 1e-5, len(x)))


@pytest.mark.parametrize("n", [1, 31, 127, 128, 129, 304 * 128 + 77])
def test_gradient_and_loss_at_block_edges(pflbm, oracle, n):
    x = _features(max(n, 64), 21)
    y = _targets(x, 22)
    with pflbm.Closure(len(x)) as c:
        c.set_samples(x, y)
        c.init_params(seed=3)
        blob = c.blob.copy()
        blob[:1377] += np.random.default_rng(4).normal(0.0, 0.05, 1377).astype(np.float32)
        c.blob = blob
        c.set_samples(x[:n], y[:n])
        g, loss = c.gradient(n)
        mean = c.loss()
    p, mu, sc, osc = _split(blob.astype(np.float64))
    x32, y32 = x[:n].astype(np.float32).astype(np.float64), y[:n].astype(np.float32).astype(np.float64)
    out, ref = oracle.mlp_eval(p, mu, sc, osc, x32, y32, with_grad=True)
    loss_ref = float(np.sum((out / osc - y32 / osc) ** 2))
    tol = 8 * 2.0 ** -11
    assert np.linalg.norm(g - ref) <= tol * np.linalg.norm(ref)
    assert loss == pytest.approx(loss_ref, rel=tol)
    assert mean == pytest.approx(loss_ref / n, rel=1e-5)


def _mix64(v):
    with np.errstate(over="ignore"):
        v = (v ^ (v >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        v = (v ^ (v >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        return v ^ (v >> np.uint64(31))


@pytest.mark.parametrize("batch", [1, 130, 16384, 304 * 128 + 200])
def test_training_iterations_are_adam_on_the_gradient(pflbm, batch):
    n, seed, lr = 50_000, 9, 2e-3
    b1, b2 = float(np.float32(0.9)), float(np.float32(0.999))
    x = _features(n, 31).astype(np.float32)
    y = _targets(x.astype(np.float64), 32).astype(np.float32)
    m, v = np.zeros(1377), np.zeros(1377)
    with pflbm.Closure(n) as c, pflbm.Closure(batch) as own:
        c.set_samples(x, y)
        c.init_params(seed=3)
        for t in range(1, 4):
            before = c.blob.copy()
            with np.errstate(over="ignore"):
                k = np.uint64(t) * np.uint64(0x100000001B3) + np.arange(batch, dtype=np.uint64)
                at = _mix64(np.uint64(seed) * np.uint64(0x9E3779B97F4A7C15) + _mix64(k)) % np.uint64(n)
            own.set_samples(x[at.astype(np.int64)], y[at.astype(np.int64)])
            own.blob = before
            g, loss = own.gradient(batch)
            history = c.train(1, batch=batch, lr=lr, seed=seed)
            m = b1 * m + (1 - b1) * g / batch
            v = b2 * v + (1 - b2) * (g / batch) ** 2
            step = lr * (m / (1 - b1 ** t)) / (np.sqrt(v / (1 - b2 ** t)) + 1e-8)
            assert np.abs(c.blob[:1377] - (before[:1377] - step)).max() <= 2.4e-7 + 1e-5 * lr
            assert history[0] == pytest.approx(loss / batch, rel=1e-6)


def test_training_in_one_call_or_many(pflbm):
    """300 iterations span several launches; the state carries over bit for bit."""
    x = _features(5000, 41)
    y = _targets(x, 42)
    blobs = []
    for calls in ((300,), (1, 128, 171)):
        with pflbm.Closure(5000) as c:
            c.set_samples(x, y)
            c.init_params(seed=3)
            hist = np.concatenate([c.train(k, batch=1000, lr=2e-3, seed=5) for k in calls])
            blobs.append((c.blob.copy(), hist))
    assert np.array_equal(blobs[0][0], blobs[1][0]) and np.array_equal(blobs[0][1], blobs[1][1])
