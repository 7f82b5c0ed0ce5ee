"""What a training run reports and where it ends, replayed on the host.

The run is replayed from the documented steps: samples and labels from the seed, the
oracle's gradients with BF16 rounding, Adam with a cosine decay. Tolerances:
 - Weights. A gradient is within 1e-3 of the oracle's (test_gpu_train_step.py derives it).
   Adam's step depends on the sign of a gradient where it is small: a share of about 1e-3 of
   the elements has one below 1e-3 of the usual size and may step the other way, which moves
   the weights by at most 2 sqrt(1e-3) = 6 % of a step; 10 % of the movement covers it. Leaving
   out one of the four steps, or misreading a partial minibatch's rows, moves them by more.
 - Loss of the replayed run. It follows the weights: 1e-2.
 - Loss of a run that does not move (a step size of 1e-30). One FP32 total over 32 steps has
   a unit in the last place of 2^-23 of 32 minibatch losses, an eighth of the mean element
   (32,768 to a minibatch). Rounding an element to it errs by up to half of that, 1/16 of the
   mean element, with either sign; only elements below the half are always lost, and they
   hold (1/16)^(3/2) / 3 = 0.5 % of a sum of squares at most."""

import ctypes as C
import math

import numpy as np
import pytest

import lambda_b200 as lb
from lambda_b200 import _native as N
from lambda_b200 import surrogate
from oracle import port

pytestmark = pytest.mark.gpu

MASK = (1 << 64) - 1


def _splitmix(x):
    x = x + np.uint64(0x9E3779B97F4A7C15)
    x = (x ^ (x >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    x = (x ^ (x >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return x ^ (x >> np.uint64(31))


def _samples(n, seed):
    """The run's inputs and labels."""
    r = lb.default_film_range()
    i = np.arange(n, dtype=np.uint64)
    q = []
    for d, k in enumerate(surrogate.RANGE_KEYS):
        lo, hi = (np.float32(v) for v in getattr(r, k))
        u = (_splitmix(np.uint64(seed) ^ _splitmix(i * np.uint64(8) + np.uint64(d))) >> np.uint64(11)).astype(np.float64)
        q.append((np.float64(lo) + np.float64(hi - lo) * (u / 9007199254740992.0)).astype(np.float32))
    q = np.stack(q, 1)
    return surrogate.encode(q, r), port.film(q).astype(np.float32)


def _start(seed):
    p, s, off = np.zeros(N.MLP_PARAMS), (seed * 0x9E3779B97F4A7C15 + 1) & MASK, 0
    for out, inp, gain in ((64, 5, 1.0), (64, 64, 1.0), (64, 64, 1.0), (4, 64, 0.5)):
        a = gain * math.sqrt(6.0 / inp)
        for k in range(out * inp):
            s = (s * 6364136223846793005 + 1442695040888963407) & MASK
            p[off + k] = np.float32(a * ((s >> 11) / 9007199254740992.0 * 2.0 - 1.0))
        off += out * inp + out
    return p


def _replay(samples, epochs, batch, lr, seed):
    x, y = _samples(samples, seed)
    p = _start(seed)
    m, v = np.zeros_like(p), np.zeros_like(p)
    steps = -(-samples // batch)
    total, t, loss = steps * epochs, 0, 0.0
    for _ in range(epochs):
        loss = 0.0
        for s in range(steps):
            rows = slice(s * batch, min(samples, (s + 1) * batch))
            l, g = port.mlp_grad(p, x[rows], y[rows], bf16=True)
            loss += l / steps
            rate = lr * (0.02 + 0.98 * 0.5 * (1 + math.cos(math.pi * t / max(1, total - 1))))
            m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
            p = p - rate * (m / (1 - 0.9 ** (t + 1))) / (np.sqrt(v / (1 - 0.999 ** (t + 1))) + 1e-8)
            t += 1
    return p, loss


@pytest.mark.parametrize("samples,batch", [(200, 128), (256, 128), (148 * 64 + 100, 148 * 64)])
def test_a_run_is_the_host_replay(ctx, samples, batch):
    """Minibatches of whole and partial slices; the last ones partial, and of more slices
    than one per SM."""
    kw = dict(samples=samples, epochs=2, batch=batch, lr=1e-3, seed=21)
    rep = ctx.surrogate_train(**kw)
    got = ctx.surrogate_get()[0]
    want, loss = _replay(**kw)
    start = _start(21)
    assert np.linalg.norm(got - want) <= 0.1 * np.linalg.norm(want - start)
    assert abs(rep.final_loss - loss) <= 1e-2 * loss


@pytest.mark.parametrize("samples,batch", [(200, 128), (262_144, 8192), (200_000, 148 * 64 * 3)])
def test_the_reported_loss_is_the_same_every_time(ctx, samples, batch):
    losses = {ctx.surrogate_train(samples=samples, epochs=1, batch=batch, lr=2e-3, seed=4).final_loss for _ in range(5)}
    assert len(losses) == 1


def test_the_reported_loss_is_near_the_mean(ctx):
    """Against the double-precision mean over the samples, at weights that do not move."""
    n, seed = 262_144, 9
    rep = ctx.surrogate_train(samples=n, epochs=1, batch=8192, lr=1e-30, seed=seed)
    x, y = _samples(n, seed)
    out = port.mlp_forward(_start(seed), x, bf16=True)
    want = float(np.mean((out - y.astype(np.float64)) ** 2))
    print(f"reported {rep.final_loss:.7g}, mean {want:.7g}: {rep.final_loss / want - 1:+.2%}")
    assert -5e-3 <= rep.final_loss / want - 1 <= 1e-3


@pytest.mark.parametrize("n", [1, 64, 65, 10_000])
@pytest.mark.parametrize("target", [1e25, -3e19, np.inf])
def test_an_infinite_loss_stays_infinite(ctx, n, target):
    """Squares beyond FP32 (or an infinite target) make the loss infinite, not NaN."""
    rng = np.random.default_rng(2)
    p = rng.normal(0, 0.3, N.MLP_PARAMS).astype(np.float32)
    x = rng.uniform(-1, 1, (n, 5)).astype(np.float32)
    y = rng.uniform(0, 1, (n, 4)).astype(np.float32)
    y[n // 2, 1] = target
    g = np.empty(N.MLP_PARAMS, np.float32)
    loss = C.c_float()
    st = ctx._lib.lambda_surrogate_grad(ctx._h, p.ctypes.data, x.ctypes.data, y.ctypes.data, n, g.ctypes.data,
                                        C.byref(loss))
    assert st == 0, ctx.last_error
    assert loss.value == math.inf
