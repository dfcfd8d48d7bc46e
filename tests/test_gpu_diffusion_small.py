"""The diffusion quotient over the whole range of magnitudes (GPU required): one sweep of fields
scaled by a power of two, against the oracle's division in double.

q = fma(num, rh, num*rl) with rh + rl = 1/D has an error below 2^-47 of the quotient before its
last rounding, and at most 2^-150 more where num*rl is no normal number: so q is at most one unit
in the last place off, and equal but for about two quotients in 2^23 while num*rl, some 2^-41 of
num at a divisor of 4e4, is well above 2^-126."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rate", [1e-6, 1e-3, 0.5])
@pytest.mark.parametrize("shift", [0, 40, 80, 96, 110, 124, 130, 145])
def test_one_sweep(fluid, rate, shift):
    n, dt = 130, 0.1
    rng = np.random.default_rng(shift)
    d = np.ldexp(rng.uniform(0.5, 1.0, (n, n)), -shift).astype(np.float32)
    z = np.zeros((n, n), np.float32)
    with fluid.Solver(n, n, diffuse_iterations=1, device=0) as s:
        s.upload(d, z, z)
        s.upload_sources(z, z, z)
        s.stage(fluid.STAGE_DIFFUSE_DENSITY, rate, dt)
        got = s.download()[0]
    want = oracle.diffuse(d, 0, rate, dt, 1)
    inner = np.s_[1:-1, 1:-1]
    off = np.abs(got[inner].view(np.int32).astype(np.int64) - want[inner].view(np.int32))
    assert off.max() <= 1
    if shift <= 80:
        assert np.count_nonzero(off) == 0
