"""The tail of the exact reductions: the last block's lanes fetch one limb each and lane 0 forms the
result from all of them. Terms in every limb (2^-158 to 2^120), one block and many, repeated: each
result is the exactly rounded sum."""
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [40, 256, 257, 16384, 200_003])
def test_every_limb_of_a_sum_is_read(ctx, stslib, n):
    rng = np.random.default_rng(n)
    a = rng.standard_normal(n) * np.exp2(rng.integers(-100, 120, size=n))
    a[:8] = np.ldexp(rng.choice([-1.0, 1.0], 8) * 1.5, [-158, -126, -94, -62, -30, 2, 34, 66])
    one = stslib.NVector.from_numpy(ctx, np.ones(n))
    for sign in (1.0, -1.0):
        b = sign * a
        # the accumulator's terms: multiples of 2^-160, truncated toward zero
        total = sum(int(Fraction(float(v)) * 2 ** 160) for v in b)
        want = float(Fraction(total, 2 ** 160))
        B = stslib.NVector.from_numpy(ctx, b)
        assert [B.dot(one) for _ in range(200)] == [want] * 200
