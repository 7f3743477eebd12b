"""Forms that only large grids take by default, bit for bit against the oracle: groups of eight mixed
stages on 112 x 48 tiles, and eight rows per thread in the periodic stages and their step end."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def one_step(ctx, stslib, oracle, pk, h, mixed):
    P, O = stslib.Problem(ctx, **pk), oracle.Problem(**pk)
    y0 = np.random.default_rng(pk["nx"]).standard_normal(P.n)
    I = stslib.LSRKStep(ctx, P, 0.0, stslib.NVector.from_numpy(ctx, y0), method=1, hfixed=h, mixed=mixed)
    J = oracle.Integrator(O, y0.copy(), method=1, rtol=1e-6, atol=1e-10, hfixed=h, mixed=mixed)
    y = P.vector()
    I.evolve(h, y)
    assert J.evolve(h) == 0
    assert I.stats()["nst"] == 1
    assert np.array_equal(y.numpy(), J.y)
    return I


# 508 and 511 tiles of 112 x 32: more than those are allowed below 1.56 million points, so 48 rows;
# 8100 rows are 36 short of whole tiles, 2305 one more; 113 and 673 columns one more than whole tiles.
# The last grid is above that size: timed, so any group size may win.
@pytest.mark.parametrize("nx,ny,config", [(113, 8100, 7), (673, 2305, 7), (1347, 1201, None)])
@pytest.mark.parametrize("kind", [0, 1])
def test_eight_stages_on_48_rows_bitwise(ctx, stslib, oracle, nx, ny, config, kind):
    pk = dict(kind=kind, nx=nx, ny=ny, kx=1.0, ky=0.3)
    h = 245.0 / (1.01 * 8.0 * max((nx + 1) ** 2, 0.3 * (ny + 1) ** 2))  # 22 stages: 1 + 8 + 8 + 4 + 1
    I = one_step(ctx, stslib, oracle, pk, h, True)
    assert I.stats()["stage_max"] == 22
    if config is not None:
        info = I.stage_fusion_info()
        assert (info["ks"], info["config"], info["tile_rows"]) == (8, config, 48)


# on both sides of ten times 1024 points per SM (1 556 480), with ragged last rows and columns
@pytest.mark.parametrize("nx,ny", [(1249, 1246), (1248, 1248), (1251, 1253), (67, 23_333)])
@pytest.mark.parametrize("inhomogeneous", [False, True])
@pytest.mark.parametrize("mixed", [False, True])
def test_periodic_rows_per_thread_bitwise(ctx, stslib, oracle, nx, ny, inhomogeneous, mixed):
    pk = dict(kind=2, nx=nx, ny=ny, kx=1.0, ky=0.3, inhomogeneous=inhomogeneous)
    h = 30.0 / (16.0 * max((nx / 6.2) ** 2, 0.3 * (ny / 12.0) ** 2))
    one_step(ctx, stslib, oracle, pk, h, mixed)
