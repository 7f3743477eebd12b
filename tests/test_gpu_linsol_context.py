"""The generic CG works in the context of its vectors, whichever context it was created with, and like a
vector it may be freed after the context."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_solver_created_with_another_context(ctx, stslib):
    other = stslib.Context(0)
    G = stslib.Problem(ctx, 0, 700, 500, 1.0, 0.1)
    gamma = 1e-4
    B = stslib.NVector.from_numpy(ctx, np.random.default_rng(5).standard_normal(G.n))
    tmp, x = G.vector(), G.vector()

    def atimes(v, z):
        G.jac_times(v, tmp)
        z.linear_sum(1.0, v, -gamma, tmp)

    def solve(c):
        S = stslib.PCGSolver(c, B, atimes, lambda r, z: G.psolve(r, z, gamma), maxl=400)
        rc, it, res = S.solve(x, B, 1e-9)
        assert rc == 0
        return x.numpy(), it, res

    y, it, res = solve(ctx)
    for _ in range(5):
        z, it2, res2 = solve(other)
        assert np.array_equal(y, z) and it == it2 and res == res2


def test_solver_freed_after_its_context(stslib):
    L = stslib.lib()
    c = C.c_void_p()
    assert L.STS_ContextCreate(0, C.byref(c)) == 0
    y = L.N_VNew_Sts(1000, c)
    S = L.STS_SUNLinSol_PCG(y, 0, 10, c)
    assert S
    assert L.STS_ContextFree(C.byref(c)) == 0
    assert L.STS_SUNLinSolFree(S) == 0
    L.N_VDestroy_Sts(y)
