"""The training step over slices of 64 rows: gradients against the FP64 oracle at row
counts on both sides of a slice, of one slice per SM and of several slices per CTA, and
a training run that ends in a partial minibatch.

Tolerance: FP32 sums of n terms err by about sqrt(n) 2^-24 relative (2e-5 at 2^17); an
activation whose FP32 sum falls on the other side of a BF16 rounding boundary than the
FP64 one moves by 2^-8, which happens to about 64 x 2^-24 / 2^-9 = 2e-3 of them at most,
so the gradient of n random rows moves by at most 2^-8 sqrt(2e-3 / n): 2e-4 at one row.
1e-3 covers both."""

import ctypes as C

import numpy as np
import pytest

import lambda_b200 as lb
from lambda_b200 import _native as N
from oracle import port

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 63, 64, 65, 127, 128, 148 * 64, 148 * 64 + 1, 20000, 65536])
def test_gradient_at_slice_boundaries(ctx, n):
    rng = np.random.default_rng(n)
    p = rng.normal(0, 0.3, N.MLP_PARAMS).astype(np.float32)
    x = rng.uniform(-1, 1, (n, 5)).astype(np.float32)
    y = rng.uniform(0, 1, (n, 4)).astype(np.float32)
    got = []
    for _ in range(2):
        g = np.empty(N.MLP_PARAMS, np.float32)
        loss = C.c_float()
        st = ctx._lib.lambda_surrogate_grad(ctx._h, p.ctypes.data, x.ctypes.data, y.ctypes.data, n, g.ctypes.data,
                                            C.byref(loss))
        assert st == 0, ctx.last_error
        got.append(g)
    assert np.array_equal(got[0], got[1])  # every sum has a fixed order
    want_loss, want = port.mlp_grad(p.astype(np.float64), x, y, bf16=True)
    rel = float(np.linalg.norm(got[0] - want) / np.linalg.norm(want))
    assert rel < 1e-3, rel
    assert abs(loss.value - want_loss) <= 1e-3 * abs(want_loss)


@pytest.mark.parametrize("samples,batch", [(64, 64), (1000, 128), (148 * 64 * 3 + 17, 148 * 64 * 2)])
def test_training_runs_with_a_partial_minibatch(ctx, samples, batch):
    kw = dict(samples=samples, epochs=2, batch=batch, lr=1e-3, seed=5, film_range=lb.default_film_range())
    a = ctx.surrogate_train(**kw)
    pa = ctx.surrogate_get()[0]
    b = ctx.surrogate_train(**kw)
    pb = ctx.surrogate_get()[0]
    assert np.array_equal(pa, pb) and np.isfinite(pa).all()
    assert np.isfinite(a.final_loss) and a.max_abs_error == b.max_abs_error
    # two epochs from the same start: weights have moved by at most lr per step and bias correction
    assert 0 < a.mean_abs_error <= a.max_abs_error
