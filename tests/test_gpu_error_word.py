"""A kernel that gives up a bounded wait sets the context's error word in mapped host memory. The word may
arrive after the step's result; evolve reports it at the latest when it returns."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def error_word(ctx):
    """STS_Context_: two ints, then stream, d_work, h_slots, d_slots, h_err."""
    return C.cast(C.cast(ctx.h, C.POINTER(C.c_void_p))[5], C.POINTER(C.c_int))


@pytest.mark.parametrize("kind,mixed", [(0, False), (0, True), (2, False), (2, True)])
def test_late_error_word_fails_the_call(ctx, stslib, kind, mixed):
    P = stslib.Problem(ctx, kind, 96, 64, 1.0, 0.1)
    I, J = (stslib.LSRKStep(ctx, P, 0.0, P.initial(), method=stslib.RKL, mixed=mixed) for _ in range(2))
    y, z = P.vector(), P.vector()
    t = 0.01 if kind == 0 else 0.1
    I.evolve(t, y)
    J.evolve(t, z)
    word = error_word(ctx)
    assert word[0] == 0
    word[0] = 1
    # (no step is left to take, so only the look after the call's synchronisation can see it)
    with pytest.raises(stslib.STSError, match="pipeline wait timed out"):
        I.evolve(t, y)
    assert word[0] == 0
    I.evolve(3 * t, y)
    J.evolve(3 * t, z)
    assert np.array_equal(y.numpy(), z.numpy())
