"""ARKodeSetUserData hands an integrator that has stepped another problem with as many points: every call
that may come next works on the new problem alone, bit for bit as an integrator created for it."""
import numpy as np
import pytest

import ceda_demonstrations_gb300 as sts

pytestmark = pytest.mark.gpu
H = 2e-4


def make(ctx, kind, nx, ny, ky=0.3):
    """A problem whose spectral radius stays below the bound that the integrators are given."""
    kx = min(1.0, 1e5 / max(nx, ny) ** 2)
    return sts.Problem(ctx, kind, nx, ny, kx, ky * kx, inhomogeneous=kind == sts.PERIODIC)


def state(ctx, P, seed=1):
    return sts.NVector.from_numpy(ctx, np.random.default_rng(seed).standard_normal(P.nx * P.ny))


def integrator(ctx, P, y0, mixed):
    """Fixed steps of the same stage count on either problem, whatever ran before."""
    return sts.LSRKStep(ctx, P, 0.0, y0, method=sts.RKL, mixed=mixed, hfixed=H, dom_eig=lambda t: -6e5)


def run(I, P, t):
    y = P.vector()
    I.set_stop_time(t)
    I.evolve(t, y)
    return y.numpy()


def switch(I, P):
    assert sts.lib().STS_ARKodeSetUserData(I.mem, P.h) == 0


# rows of the first shape need no padding in the FP32 fields, of the second two or three columns
SHAPES = [((40, 21), (42, 20)), ((120, 70), (105, 80)), ((1200, 700), (1050, 800))]


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("shapes", SHAPES, ids=str)
def test_another_shape_then_reset(ctx, shapes, mixed):
    A, B = (make(ctx, sts.MANUFACTURED, *s) for s in shapes)
    I = integrator(ctx, A, state(ctx, A), mixed)
    ya = run(I, A, 2 * H)
    y1 = state(ctx, B, 2)
    switch(I, B)
    I.reset(0.0, y1)
    assert np.array_equal(run(I, B, 3 * H), run(integrator(ctx, B, y1, mixed), B, 3 * H))
    switch(I, A)  # and back
    I.reset(0.0, state(ctx, A))
    assert np.array_equal(run(I, A, 2 * H), ya)


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("shapes", SHAPES, ids=str)
def test_another_shape_then_checkpoint(ctx, tmp_path, shapes, mixed):
    A, B = (make(ctx, sts.MANUFACTURED, *s) for s in shapes)
    # reading one
    J = integrator(ctx, B, state(ctx, B, 2), mixed)
    run(J, B, 2 * H)
    J.write_checkpoint(str(tmp_path / "b"))
    yb = run(J, B, 4 * H)
    I = integrator(ctx, A, state(ctx, A), mixed)
    run(I, A, 2 * H)
    switch(I, B)
    I.read_checkpoint(str(tmp_path / "b"))
    assert np.array_equal(run(I, B, 4 * H), yb)
    # writing one: it holds what the integrator continues from
    K = integrator(ctx, A, state(ctx, A), mixed)
    run(K, A, 2 * H)
    switch(K, B)
    K.write_checkpoint(str(tmp_path / "k"))
    L = integrator(ctx, B, state(ctx, B, 2), mixed)
    L.read_checkpoint(str(tmp_path / "k"))
    assert np.array_equal(run(K, B, 4 * H), run(L, B, 4 * H))


@pytest.mark.parametrize("mixed", [False, True])
def test_stage_timing_after_a_change_and_a_checkpoint(ctx, tmp_path, mixed):
    A, B = make(ctx, sts.MANUFACTURED, 120, 70), make(ctx, sts.MANUFACTURED, 105, 80)
    I = integrator(ctx, A, state(ctx, A), mixed)
    run(I, A, 2 * H)
    I.write_checkpoint(str(tmp_path / "a"))
    want = run(I, A, 4 * H)
    J = integrator(ctx, A, state(ctx, A), mixed)
    J.read_checkpoint(str(tmp_path / "a"))
    assert J.time_stage_kernel(3) > 0.0  # no stage has run in this integrator
    assert np.array_equal(run(J, A, 4 * H), want)
    switch(I, B)
    assert I.time_stage_kernel(3) > 0.0
    y1 = state(ctx, B, 2)
    I.reset(0.0, y1)
    assert np.array_equal(run(I, B, 3 * H), run(integrator(ctx, B, y1, mixed), B, 3 * H))


SAME = [(sts.MANUFACTURED, 0.3, sts.MANUFACTURED, 0.05), (sts.MANUFACTURED, 0.3, sts.UNFORCED, 0.3),
        (sts.UNFORCED, 0.1, sts.MANUFACTURED, 0.2), (sts.PERIODIC, 0.3, sts.PERIODIC, 0.05)]


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("case", SAME, ids=str)
def test_same_shape_other_coefficients_or_kind(ctx, case, mixed):
    """Steps recorded for one problem, and the FP32 faces of a periodic one, are not used for another."""
    A, B = make(ctx, case[0], 120, 70, case[1]), make(ctx, case[2], 120, 70, case[3])
    I = integrator(ctx, A, state(ctx, A), mixed)
    ya = run(I, A, 3 * H)
    y1 = state(ctx, B, 2)
    switch(I, B)
    I.reset(0.0, y1)
    assert np.array_equal(run(I, B, 3 * H), run(integrator(ctx, B, y1, mixed), B, 3 * H))
    switch(I, A)
    I.reset(0.0, state(ctx, A))
    assert np.array_equal(run(I, A, 3 * H), ya)


@pytest.mark.parametrize("mixed", [False, True])
def test_periodic_problem_of_another_shape(ctx, mixed):
    A, B = make(ctx, sts.PERIODIC, 105, 80), make(ctx, sts.PERIODIC, 84, 100)
    I = integrator(ctx, A, state(ctx, A), mixed)
    run(I, A, 2 * H)
    y1 = state(ctx, B, 2)
    switch(I, B)
    I.reset(0.0, y1)
    assert np.array_equal(run(I, B, 3 * H), run(integrator(ctx, B, y1, mixed), B, 3 * H))


# the periodic problem keeps its state elsewhere than the Dirichlet ones; 105 columns need padding
ORDERS = [(sts.PERIODIC, (105, 80), sts.MANUFACTURED, (105, 80)), (sts.MANUFACTURED, (105, 80), sts.PERIODIC, (84, 100)),
          (sts.PERIODIC, (84, 100), sts.UNFORCED, (105, 80))]


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("order", ORDERS, ids=str)
def test_between_periodic_and_dirichlet(ctx, tmp_path, order, mixed):
    A, B = make(ctx, order[0], *order[1]), make(ctx, order[2], *order[3])
    I = integrator(ctx, A, state(ctx, A), mixed)
    ya = run(I, A, 2 * H)
    y1 = state(ctx, B, 2)
    switch(I, B)
    I.reset(0.0, y1)
    J = integrator(ctx, B, y1, mixed)
    assert np.array_equal(run(I, B, 2 * H), run(J, B, 2 * H))
    I.write_checkpoint(str(tmp_path / "i"))
    K = integrator(ctx, B, state(ctx, B, 3), mixed)
    K.read_checkpoint(str(tmp_path / "i"))
    assert np.array_equal(run(K, B, 4 * H), run(J, B, 4 * H))
    switch(I, A)
    I.reset(0.0, state(ctx, A))
    assert np.array_equal(run(I, A, 2 * H), ya)
    switch(I, B)
    I.read_checkpoint(str(tmp_path / "i"))
    assert np.array_equal(run(I, B, 4 * H), run(integrator_from(ctx, B, tmp_path / "i", mixed), B, 4 * H))


def integrator_from(ctx, P, path, mixed):
    I = integrator(ctx, P, state(ctx, P, 3), mixed)
    I.read_checkpoint(str(path))
    return I


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("order", ORDERS, ids=str)
def test_the_state_goes_along(ctx, order, mixed):
    """Without a reset the new problem goes on from y_n: its dense output of the last step is the old
    one's, and back at the old problem the run continues as if it had not been left."""
    A, B = make(ctx, order[0], *order[1]), make(ctx, order[2], *order[3])
    I, J = (integrator(ctx, A, state(ctx, A), mixed) for _ in range(2))
    y = A.vector()
    for K in (I, J):
        K.evolve(2.5 * H, y)  # dense output within the third step
    mid = y.numpy()
    switch(I, B)
    yb = B.vector()
    assert I.evolve(2.5 * H, yb)[0] == 2.5 * H and np.array_equal(yb.numpy(), mid)
    switch(I, A)
    assert np.array_equal(run(I, A, 6 * H), run(J, A, 6 * H))
    switch(I, B)
    assert np.isfinite(run(I, B, 9 * H)).all()


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("kind", [sts.MANUFACTURED, sts.PERIODIC])
def test_another_number_of_points_is_refused(ctx, tmp_path, kind, mixed):
    """A problem larger or smaller than the state: an error before any kernel runs, and the run goes on
    with the right problem as if nothing had been asked."""
    A = make(ctx, kind, 105, 80)
    y0 = state(ctx, A)
    want = run(integrator(ctx, A, y0, mixed), A, 4 * H)
    I = integrator(ctx, A, y0, mixed)
    run(I, A, 2 * H)
    y = A.vector()
    for other in ((105, 81), (104, 80), (210, 160)):
        for k in (sts.MANUFACTURED, sts.PERIODIC):
            B = make(ctx, k, *other)
            switch(I, B)
            for call in (lambda: I.evolve(4 * H, y), lambda: I.reset(0.0, y0),
                         lambda: I.write_checkpoint(str(tmp_path / "c"))):
                with pytest.raises(sts.STSError):
                    call()
    switch(I, A)
    assert np.array_equal(run(I, A, 4 * H), want)
    B = make(ctx, kind, 104, 80)
    F = sts.LSRKStep(ctx, A, 0.0, state(ctx, B), mixed=mixed)  # from the start
    with pytest.raises(sts.STSError):
        F.evolve(H, B.vector())
