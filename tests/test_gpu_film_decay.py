"""FP64 film queries whose film is evanescent, over decays and growths (negative thickness
or wavelength) from nothing to beyond the range of the closed form, against the oracle's
complex matrices. Tolerance: both sides round about 100 operations, 1e-14; the denominator
|1 + r01 r12 e| can be small against its terms, which loses up to its inverse: 1e-9 of
the largest value covers 1e5."""

import numpy as np
import pytest

from oracle import port

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sign", [(1, 1), (1, -1), (-1, 1), (-1, -1)])
@pytest.mark.parametrize("phase", [(0, 50), (150, 250), (250, 400), (400, 650), (590, 610)])
def test_evanescent_films(ctx, sign, phase):
    r = np.random.default_rng(7)
    n = 20_000
    lam, nf = r.uniform(360, 830, n), r.uniform(0.3, 0.9, n)
    c0 = np.sqrt(1 - nf * nf) * r.uniform(0.05, 0.9, n)  # past the film's critical angle
    kappa = np.sqrt((1 - c0 * c0) / (nf * nf) - 1)
    d = r.uniform(*phase, n) / (4 * np.pi * nf * kappa / lam)  # |phase| in the range
    q = np.stack([sign[0] * lam, c0, sign[1] * d, nf, r.uniform(0.3, 2.0, n)], 1).astype(np.float32)
    got, want = ctx.thinfilm_fp64(q), port.film(q)
    assert np.array_equal(np.isfinite(got), np.isfinite(want))
    fine = np.isfinite(want)
    assert fine.any()
    assert np.abs(got - want)[fine].max() <= 1e-9 * max(1.0, np.abs(want[fine]).max())
