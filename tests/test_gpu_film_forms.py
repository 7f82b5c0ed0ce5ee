"""The FP64 film's closed form against the oracle's complex matrices, over real and
evanescent cosines in the film and the substrate and at the edges where the general
product is taken; and FP32 queries four to a thread against one to a thread, around the
size where the former starts, for partial fours and for pointers off 16 bytes.

Tolerance of the FP64 comparison: both sides round about 100 operations, 100 x 2^-53 =
1e-14 relative; past a critical angle the denominator |1 + r01 r12 e| can be small
against its terms, which loses up to its inverse: 1e-9 of the largest value covers 1e5."""

import numpy as np
import pytest

import lambda_b200 as lb
from oracle import port

pytestmark = pytest.mark.gpu


def _queries(n, seed, n_film, n_sub):
    r = np.random.default_rng(seed)
    return np.stack([r.uniform(360, 830, n), r.uniform(0, 1, n), r.uniform(0, 2000, n), r.uniform(*n_film, n),
                     r.uniform(*n_sub, n)], 1).astype(np.float32)


@pytest.mark.parametrize("name,n_film,n_sub", [
    ("no critical angle", (1.0, 2.5), (1.0, 3.0)),
    ("substrate past critical", (1.0, 2.5), (0.3, 1.0)),
    ("film past critical", (0.4, 1.0), (1.0, 3.0)),
    ("both past critical", (0.4, 1.0), (0.3, 1.0)),
])
def test_fp64_closed_form_matches_the_complex_product(ctx, name, n_film, n_sub):
    q = _queries(20000, 3, n_film, n_sub)
    q[:20, 1] = 1.0           # normal incidence
    q[20:40, 2] = 0.0         # no film
    q[40:60, 3] = q[40:60, 4]  # film like the substrate
    q[60:80, 3] = 1.0         # film like the outer medium
    got, want = ctx.thinfilm_fp64(q), port.film(q)
    assert np.array_equal(np.isfinite(got), np.isfinite(want))
    fine = np.isfinite(want)
    assert np.abs(got - want)[fine].max() <= 1e-9 * max(1.0, np.abs(want[fine]).max())


@pytest.mark.parametrize("n", [(1 << 20) - 1, 1 << 20, (1 << 20) + 1, (1 << 20) + 3])
@pytest.mark.parametrize("offset", [0, 1])
def test_four_queries_per_thread_give_the_same_bits(ctx, n, offset):
    import torch

    q = _queries(n, 9, (1.2, 1.8), (1.0, 2.0))
    buf = torch.zeros(5 * n + offset, dtype=torch.float32, device="cuda")
    buf[offset:] = torch.from_numpy(q).reshape(-1).cuda()
    dq = buf[offset:].view(n, 5)
    out = torch.full((n, 4), -1.0, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    ctx.thinfilm_exact(dq, out)
    got = out.cpu().numpy()
    for a in range(0, n, 500_000):  # below the size where a thread takes four
        want = ctx.thinfilm_exact(q[a:a + 500_000])
        assert np.array_equal(got[a:a + 500_000].view(np.uint32), want.view(np.uint32))
