"""Results that the host polls for in mapped slots: a call that returns an error leaves no reduction in
flight whose late result a later call could take for its own."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_dot_products_after_a_refused_call(ctx, stslib):
    n = 2_000_000
    new = stslib.NVector.from_numpy
    one, two, three = (new(ctx, np.full(n, v)) for v in (1.0, 2.0, 3.0))
    short = new(ctx, np.ones(n - 1))
    for _ in range(20):
        for k in range(1, 48, 7):
            with pytest.raises(stslib.STSError):
                one.dot_multi([two] * k + [short])
            assert list(one.dot_multi([three] * k)) == [3.0 * n] * k
    with pytest.raises(stslib.STSError):
        one.dot_multi([short])
    assert list(one.dot_multi([two])) == [2.0 * n]
