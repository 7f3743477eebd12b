"""Learned multilevel preconditioner: GPU forward/backward kernels against the FP64 CPU
reference (oracle/convnet.py), batched training, and flexible CG with the trained network
against Jacobi-PCG on the same shifted systems (I - gamma A) x = b.

Tolerances: the GPU keeps weights and activations in BF16 (8-bit mantissa, relative
rounding 2^-9 per stored value) with FP32 accumulation, the reference computes in FP64 from
the same BF16 weights; nine stored layers give a few 1e-3 relative error, so the forward
output is held to 3e-2 relative L2 and each layer's weight gradient to 6e-2.
"""
import numpy as np
import pytest

import ceda_demonstrations_gb300 as sts
from oracle import convnet

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

FWD_TOL = 3e-2
GRAD_TOL = 6e-2


def _rel(a, b):
    return float(np.linalg.norm(np.ravel(a) - np.ravel(b)) / np.linalg.norm(np.ravel(b)))


def _f32_dev(a):
    t = torch.as_tensor(np.ascontiguousarray(a, dtype=np.float32)).cuda()
    torch.cuda.synchronize()
    return t


def _smooth_field(n, rng):
    return sts.smooth_field(n, rng)


@pytest.fixture(scope="module")
def weights():
    return convnet.init_weights(seed=3)


@pytest.mark.parametrize("n,sk,sg", [(64, 0.3, -0.5), (128, -1.0, 0.8)])
def test_forward_matches_oracle(ctx, weights, n, sk, sg):
    rng = np.random.default_rng(n)
    r = rng.standard_normal((n, n))
    jac = 0.37
    net = sts.Net(ctx, 128, seed=0)
    net.set_weights(weights)
    rv = sts.NVector.from_numpy(ctx, r)
    zv = sts.NVector(ctx, n * n)
    net.apply(n, rv.ptr, zv.ptr, sk, sg, jac, 1.0)
    z = zv.numpy().reshape(n, n)
    zref, _ = convnet.forward(weights, r, sk, sg, jac)
    assert _rel(z, zref) < FWD_TOL
    # power-of-two input scaling commutes with every BF16 rounding: bitwise identical output
    net.apply(n, rv.ptr, zv.ptr, sk, sg, jac, 4.0)
    assert np.array_equal(zv.numpy().reshape(n, n), z)


@pytest.mark.parametrize("n", [128, 384])
def test_tcgen05_and_mma_sync_paths_agree(ctx, weights, n):
    """The inference convolutions on tcgen05 (TMEM accumulators, 128-pixel UMMA tiles) and
    on mma.sync compute the same network: both within the oracle tolerance, and within BF16
    rounding of each other (the accumulation order inside the tensor cores differs)."""
    rng = np.random.default_rng(n + 1)
    r = rng.standard_normal((n, n))
    net = sts.Net(ctx, 384, seed=0)
    net.set_weights(weights)
    rv = sts.NVector.from_numpy(ctx, r)
    zv = sts.NVector(ctx, n * n)
    out = []
    for path in (1, 0):
        net.set_tensor_path(path)
        net.apply(n, rv.ptr, zv.ptr, 0.4, -0.2, 0.5, 1.0)
        out.append(zv.numpy().reshape(n, n))
    zref, _ = convnet.forward(weights, r, 0.4, -0.2, 0.5)
    assert _rel(out[0], zref) < FWD_TOL and _rel(out[1], zref) < FWD_TOL
    assert _rel(out[0], out[1]) < 1e-2


@pytest.mark.parametrize("n", [64, 128, 384])
def test_collapsed_level0_matches_layers(ctx, weights, n):
    """Level 0 collapsed into two kernels (stride-2 4x4 convolution for p0; 5x5 convolution
    with edge corrections plus coarse-parity kernels for z) is the same network as the
    layer-by-layer kernels: both within the oracle tolerance, within BF16 rounding of each
    other, and the collapsed form (no BF16 rounding of the fine-level tensors) closer to the
    FP64 reference."""
    rng = np.random.default_rng(n + 7)
    r = rng.standard_normal((n, n))
    net = sts.Net(ctx, 384, seed=0)
    net.set_weights(weights)
    rv = sts.NVector.from_numpy(ctx, r)
    zv = sts.NVector(ctx, n * n)
    out = []
    for on in (True, False):
        net.set_collapsed_level0(on)
        net.apply(n, rv.ptr, zv.ptr, -0.4, 0.7, 0.6, 1.0)
        out.append(zv.numpy().reshape(n, n))
    zref, _ = convnet.forward(weights, r, -0.4, 0.7, 0.6)
    e_col, e_lay = _rel(out[0], zref), _rel(out[1], zref)
    assert e_col < FWD_TOL and e_lay < FWD_TOL and e_col <= e_lay
    assert _rel(out[0], out[1]) < 1e-2


def test_weights_round_trip(ctx, weights):
    net = sts.Net(ctx, 64, seed=1)
    net.set_weights(weights)
    got = net.weights()
    for nm in convnet.NAMES:
        co, ci = convnet.shape(nm)[:2]
        assert np.array_equal(got[nm][:co, :ci], weights[nm])
        assert not np.any(got[nm][co:]) and not np.any(got[nm][:, ci:])


def test_gradients_match_oracle(ctx, weights):
    n = 64
    rng = np.random.default_rng(11)
    r = rng.standard_normal((n, n))
    e = rng.standard_normal((n, n)).astype(np.float32)
    sk, sg, jac, gcx, gcy = 0.4, -0.2, 0.5, 24.0, 3.0
    net = sts.Net(ctx, n, seed=0)
    net.set_weights(weights)
    rv = sts.NVector.from_numpy(ctx, r)
    et = _f32_dev(e)
    loss, grad = net.loss_grad(n, rv.ptr, et.data_ptr(), sk, sg, jac, gcx, gcy)
    lref, gref = convnet.loss_and_grad(weights, r, e.astype(np.float64), sk, sg, jac, gcx, gcy)
    assert abs(loss - lref) / lref < FWD_TOL
    for nm in convnet.NAMES:
        co, ci = convnet.shape(nm)[:2]
        assert _rel(grad[nm][:co, :ci], gref[nm]) < GRAD_TOL, nm
        # padded channels stay exactly zero
        assert not np.any(grad[nm][co:]) and not np.any(grad[nm][:, ci:])


@pytest.mark.parametrize("n", [16, 48, 144])
def test_gradients_on_partial_tiles(ctx, weights, n):
    """Sizes whose levels end inside a 16 x 16 tile (n/8 = 2, 6, 18), against the oracle with the
    tolerance above; sums are taken in a fixed order, so a second call gives the same bits."""
    rng = np.random.default_rng(n)
    r = rng.standard_normal((n, n))
    e = rng.standard_normal((n, n)).astype(np.float32)
    net = sts.Net(ctx, n, seed=0)
    net.set_weights(weights)
    rv, et = sts.NVector.from_numpy(ctx, r), _f32_dev(e)
    args = (n, rv.ptr, et.data_ptr(), 0.4, -0.2, 0.5, 24.0, 3.0)
    _, grad = net.loss_grad(*args)
    _, again = net.loss_grad(*args)
    _, gref = convnet.loss_and_grad(weights, r, e.astype(np.float64), 0.4, -0.2, 0.5, 24.0, 3.0)
    for nm in convnet.NAMES:
        co, ci = convnet.shape(nm)[:2]
        assert _rel(grad[nm][:co, :ci], gref[nm]) < GRAD_TOL, nm
        assert np.array_equal(grad[nm], again[nm])


def _harvest(ctx, n, ky, gam_rel, crop, ncrops, every, max_pairs, seed):
    p = sts.Problem(ctx, sts.UNFORCED, n, n, 1.0, ky)
    dx = 1.0 / (n + 1)
    gamma = gam_rel * dx * dx
    b = sts.NVector.from_numpy(ctx, _smooth_field(n, np.random.default_rng(seed)))
    r_t = torch.empty(max_pairs * crop * crop, dtype=torch.float32, device="cuda")
    e_t = torch.empty_like(r_t)
    meta = torch.empty(max_pairs * 7, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    npairs, iters = sts.harvest_pcg_pairs(p, gamma, b, ncrops, crop, every, max_pairs,
                                          r_t.data_ptr(), e_t.data_ptr(), meta.data_ptr(), seed)
    r_t = r_t[:npairs * crop * crop].view(npairs, -1)
    e_t = e_t[:npairs * crop * crop].view(npairs, -1)
    meta = meta[:npairs * 7].view(npairs, 7)
    torch.cuda.synchronize()
    return p, b, gamma, r_t, e_t, meta, iters


def test_harvest_pairs_satisfy_the_system(ctx):
    """Away from the crop edges, (I - gamma A) e_k = r_k holds for every harvested pair."""
    n, crop = 128, 64
    p, b, gamma, r_t, e_t, meta, iters = _harvest(ctx, n, 0.3, 300.0, crop, 2, 2, 16, 5)
    assert r_t.shape[0] == 16 and iters > 16
    dx = 1.0 / (n + 1)
    # metadata: features of the system, 1/rms(r) and 1/(e^T M e) of each crop
    sk, sg, jac, gcx, gcy = sts.net_features(1.0, 0.3, gamma, dx)
    m = meta.double().cpu().numpy()
    assert np.allclose(m[:, [0, 1, 2, 5, 6]], [sk, sg, jac, gcx, gcy], rtol=1e-6)
    r0 = r_t[0].double().cpu().numpy().reshape(crop, crop)
    e0 = e_t[0].double().cpu().numpy().reshape(crop, crop)
    assert np.isclose(m[0, 3], 1.0 / np.sqrt(np.mean(r0 ** 2)), rtol=1e-5)
    assert np.isclose(m[0, 4], 1.0 / np.sum(e0 * convnet.apply_M(e0, gcx, gcy)), rtol=1e-5)
    cx, cy = 1.0 / dx ** 2, 0.3 / dx ** 2
    for k in range(4):
        e = e_t[k].double().cpu().numpy().reshape(crop, crop)
        r = r_t[k].double().cpu().numpy().reshape(crop, crop)
        lap = cx * (e[1:-1, :-2] + e[1:-1, 2:]) + cy * (e[:-2, 1:-1] + e[2:, 1:-1]) \
            - 2 * (cx + cy) * e[1:-1, 1:-1]
        res = e[1:-1, 1:-1] - gamma * lap
        # e is stored in FP32: its rounding, amplified by gamma * 4 / dx^2, bounds the error
        scale = np.abs(e).max() * (1 + 4 * gamma * (cx + cy))
        assert np.abs(res - r[1:-1, 1:-1]).max() < 1e-5 * scale


@pytest.fixture(scope="module")
def trained(ctx):
    """A network trained on pairs harvested from Jacobi-PCG solves of three 256^2 systems:
    (net, loss before, loss after)."""
    n, crop = 256, 64
    rs, es, ms = [], [], []
    for k, (ky, grel) in enumerate([(1.0, 2000.0), (0.1, 800.0), (0.01, 3000.0)]):
        _, _, _, r_t, e_t, meta, _ = _harvest(ctx, n, ky, grel, crop, 8, 4, 512, 100 + k)
        rs.append(r_t)
        es.append(e_t)
        ms.append(meta)
    r_all = torch.cat(rs).contiguous()
    e_all = torch.cat(es).contiguous()
    m_all = torch.cat(ms).contiguous()
    torch.cuda.synchronize()
    net = sts.Net(ctx, n, seed=7)
    npairs = r_all.shape[0]
    loss0 = net.train(crop, npairs, r_all.data_ptr(), e_all.data_ptr(), m_all.data_ptr(),
                      epochs=1, batch=16, lr=0.0, seed=1)
    loss = net.train(crop, npairs, r_all.data_ptr(), e_all.data_ptr(), m_all.data_ptr(),
                     epochs=30, batch=16, lr=2e-3, seed=2)
    return net, loss0, loss


def test_trained_network_cuts_fcg_iterations(ctx, trained):
    """Train on pairs harvested from Jacobi-PCG solves of three systems, then solve a fourth
    (unseen right-hand side) with FCG + network and with Jacobi-PCG to the same 1e-8 residual."""
    net, loss0, loss = trained
    n = 256
    assert loss < loss0  # the training loop lowers the energy-norm loss

    ky, grel = 0.3, 1500.0
    p = sts.Problem(ctx, sts.UNFORCED, n, n, 1.0, ky)
    dx = 1.0 / (n + 1)
    gamma = grel * dx * dx
    b = sts.NVector.from_numpy(ctx, _smooth_field(n, np.random.default_rng(999)))
    x_pcg = p.vector()
    it_pcg, rel_pcg, rc = sts.implicit_solve_pcg(p, gamma, b, x_pcg, tol=1e-8)
    assert rc == 0 and rel_pcg <= 1e-8
    x_fcg = p.vector()
    it_fcg, rel_fcg, rc = sts.fcg_solve(p, gamma, net, b, x_fcg, tol=1e-8, maxit=2000)
    assert rc == 0
    assert rel_fcg <= 2e-8  # true FP64 residual of the returned iterate
    assert _rel(x_fcg.numpy(), x_pcg.numpy()) < 1e-6
    assert it_fcg < 0.5 * it_pcg, (it_fcg, it_pcg)


def test_network_as_psolve_in_flexible_gmres(ctx, trained):
    """The trained network behind the PSetup / PSolve interface (STS_NetPrec) inside
    SUNLinSol_SPFGMR, against the same solver with the Jacobi PSolve: both reach the 1e-8
    residual on an unseen system (checked on the true FP64 residual), the network in far
    fewer iterations."""
    net = trained[0]
    n, ky, grel = 256, 0.3, 1500.0
    p = sts.Problem(ctx, sts.UNFORCED, n, n, 1.0, ky)
    dx = 1.0 / (n + 1)
    gamma = grel * dx * dx
    bh = np.ascontiguousarray(_smooth_field(n, np.random.default_rng(4242)), dtype=np.float64).ravel()
    b = sts.NVector.from_numpy(ctx, bh)
    P = sts.NetPrec(net, p)
    P.setup(gamma)
    its = {}
    for name in ("net", "jacobi"):
        S = sts.SPFGMRSolver(ctx, b, maxl=40, max_restarts=300, gstype=sts.CLASSICAL_GS,
                             precond=True)
        x = p.vector()
        if name == "net":
            rc, it, res = sts.implicit_solve_ls(p, gamma, S, b, x, tol=1e-8, prec=sts.PREC_USER,
                                                pdata=P.h, psolve=P.psolve_fn)
        else:
            rc, it, res = sts.implicit_solve_ls(p, gamma, S, b, x, tol=1e-8, prec=sts.PREC_JACOBI)
        assert rc == 0 and res <= 1e-8, (name, rc, res)
        ax = p.vector()
        p.jac_times(x, ax)
        true = np.linalg.norm(bh - (x.numpy() - gamma * ax.numpy())) / np.linalg.norm(bh)
        assert true <= 2e-8, (name, true)
        its[name] = it
    assert its["net"] < 0.5 * its["jacobi"], its
    # the ARKLsPrecSolveFn form applies the same operator
    r = sts.NVector.from_numpy(ctx, bh)
    z1, z2 = p.vector(), p.vector()
    P.psolve(r, z1, gamma)
    P.psolve(r, z2, gamma)
    assert np.array_equal(z1.numpy(), z2.numpy()) and np.all(np.isfinite(z1.numpy()))


def test_sdirk2_with_learned_solves_matches_jacobi(ctx):
    """SDIRK2 on the manufactured problem with its stage systems solved by the learned-or-Jacobi
    solve (kappa ~ 7.7e3 here: the network path) agrees with the Jacobi-PCG driver to the
    solver tolerance."""
    n = 256
    P = sts.Problem(ctx, sts.MANUFACTURED, n, n, 1.0, 1.0)
    net = sts.Net(ctx, n, seed=3)
    ya, yb = P.initial(), P.initial()
    ia = sts.sdirk2_evolve(P, ya, 0.0, 0.05, 3, tol=1e-10)
    ib = sts.sdirk2_evolve_learned(P, net, yb, 0.0, 0.05, 3, tol=1e-10)
    assert ia > 0 and ib > 0
    assert _rel(yb.numpy(), ya.numpy()) < 1e-8
