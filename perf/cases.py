"""Performance cases: what programs built on this package have it compute, through its public
entry points, over the range of sizes and options that they use.

Each case is a dict with a "kind" (one of the functions' sections below) and plain parameters:

  solve    a whole small adaptive STS integration, from creating the integrator to the final
           field: the serial 128^2 configuration, and what the command-line driver does
  sts      steps of the super-time-stepping integrator on the Dirichlet problems (manufactured
           forcing or none), FP64 or mixed, RKC2 or RKL2, the stage count set by the step size
  refmode  the same integrator on the reference's periodic problem with variable coefficients,
           whose accuracy-limited steps take few stages
  batch    many independent problems of uneven sizes in one launch, host state in and out
  pcg      one shifted implicit solve (I - gamma A) x = b by Jacobi-PCG
  pfmg     the same by CG with the structured multigrid preconditioner, its setup included
  learned  iterations of flexible CG with the convolutional preconditioner (inference)
  train    one epoch of that network's training (forward, backward, Adam)
  dirk     a whole adaptive implicit DIRK integration with Newton and a Krylov solver
  nvector  the vector operations of one step of a user's own integrator

Sizes are those of the benchmark, the tests and the harness's grids, or generic ones between.
"""
import math

import numpy as np
import torch

import ceda_demonstrations_gb300 as sts

_shared = {}


def _context():
    """One library context for the whole program, as a user's program keeps one."""
    if "ctx" not in _shared:
        _shared["ctx"] = sts.Context(0)
    return _shared["ctx"]


def _wrap(ctx, t):
    """An N_Vector over the memory of a CUDA tensor (N_VMake)."""
    return sts.NVector(ctx, handle=sts.lib().N_VMake_Sts(t.numel(), t.data_ptr(), ctx.h))


# ---------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------
def listed():
    return [
        # the serial configuration of the demonstration: 128^2, RKC2, rtol 1e-6, every step
        # waits for its error norm; launches and latency are all it costs
        dict(name="solve_f64_128", kind="solve", nx=128, ny=128, kx=1.0, ky=1.0, method="rkc", mixed=False, tf=0.25),
        # FP64 field-parity configuration: 4096^2, RKL2, long stage chains
        dict(name="sts_f64_4096", kind="sts", nx=4096, ny=4096, kx=1.0, ky=1.0, forced=True, method="rkl",
             mixed=False, stages=100, steps=1),
        # the headline configuration: 8192^2 anisotropic, mixed precision, steps at the stage cap
        dict(name="sts_mixed_8192", kind="sts", nx=8192, ny=8192, kx=1.0, ky=1e-2, forced=True, method="rkl",
             mixed=True, stages=196, steps=1),
        # an ordinary mixed run on a grid whose rows are odd (no vector width divides them)
        dict(name="sts_mixed_1021x1500", kind="sts", nx=1021, ny=1500, kx=1.0, ky=0.1, forced=True, method="rkc",
             mixed=True, stages=60, steps=2),
        # the reference's own problem: periodic, coefficients k (1 + 0.99 sin), few stages a step
        dict(name="refmode_f64_1000x768", kind="refmode", nx=1000, ny=768, kx=1.0, ky=0.5, inhom=True, method="rkl",
             mixed=False, stages=9, steps=8),
        # a parameter study: independent problems of uneven sizes in one persistent launch
        dict(name="batch_f64_256", kind="batch", count=256, mixed=False, tf=2e-4),
        # implicit comparator: Jacobi-PCG on a medium, non-square grid
        dict(name="pcg_1000x700", kind="pcg", nx=1000, ny=700, ky=0.1, gamma=1e-3),
        # implicit comparator with multigrid at the implicit configuration's size
        dict(name="pfmg_2048", kind="pfmg", nx=2048, ny=2048, ky=0.05, gamma=2e-3, relax=2),
        # the learned preconditioner inside flexible CG at the implicit configuration's size
        dict(name="learned_2048", kind="learned", n=2048, ky=0.1, gamma=1e-3, iters=24),
        # training it on 128^2 residual/correction crops, minibatches of 32
        dict(name="train_128", kind="train", n=128, samples=256, batch=32),
        # the harness's default integrator on its periodic problem: DIRK, Newton, CG + Jacobi
        dict(name="dirk_128", kind="dirk", nx=128, ny=128, order=3, ls="cg", prec="jacobi", tf=0.1),
        # the smallest calls: one step's vector operations at 128^2, reductions read by the host
        dict(name="nvector_16k", kind="nvector", n=128 * 128),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "sts", "sts", "sts", "refmode", "batch", "pcg", "pfmg", "learned", "train", "dirk",
                       "nvector"])
    if kind == "solve":
        return dict(kind=kind, nx=_log(rng, 33, 200), ny=_log(rng, 33, 200), kx=1.0, ky=round(rng.uniform(0.1, 1.0), 3),
                    method=rng.choice(["rkc", "rkl"]), mixed=rng.random() < 0.4, tf=round(rng.uniform(0.05, 0.15), 3))
    if kind == "sts":
        mixed = rng.random() < 0.6
        top = 8192 if mixed else 4096
        nx, ny = _log(rng, 64, top), _log(rng, 64, top)
        if rng.random() < 0.5:
            nx -= nx % 4
        stages = _log(rng, 8, 190)
        most = (1.2e10 if mixed else 1.5e9) / (nx * ny)  # stages in all, so that a drawn case costs no more than a listed one
        stages = max(4, min(stages, int(most)))
        return dict(kind=kind, nx=nx, ny=ny, kx=1.0, ky=round(10 ** rng.uniform(-2, 0), 4),
                    forced=rng.random() < 0.6, method=rng.choice(["rkc", "rkl"]), mixed=mixed, stages=stages,
                    steps=max(1, min(rng.randint(1, 4), int(most / stages))))
    if kind == "refmode":
        return dict(kind=kind, nx=_log(rng, 64, 2048), ny=_log(rng, 64, 2048), kx=1.0,
                    ky=round(rng.uniform(0.1, 1.0), 3), inhom=rng.random() < 0.7,
                    method=rng.choice(["rkc", "rkl"]), mixed=rng.random() < 0.5, stages=rng.randint(5, 24),
                    steps=rng.randint(1, 6))
    if kind == "batch":
        return dict(kind=kind, count=_log(rng, 16, 256), mixed=rng.random() < 0.5, tf=round(10 ** rng.uniform(-4.3, -3.7), 7))
    if kind == "pcg":
        return dict(kind=kind, nx=_log(rng, 100, 1500), ny=_log(rng, 100, 1500), ky=round(10 ** rng.uniform(-3, 0), 5),
                    gamma=round(10 ** rng.uniform(-4, -2.5), 7))
    if kind == "pfmg":
        return dict(kind=kind, nx=_log(rng, 64, 2048), ny=_log(rng, 64, 2048), ky=round(10 ** rng.uniform(-3, 0), 5),
                    gamma=round(10 ** rng.uniform(-4, -2), 7), relax=rng.choice([1, 2]))
    if kind == "learned":
        return dict(kind=kind, n=16 * _log(rng, 12, 128), ky=round(10 ** rng.uniform(-3, 0), 5),
                    gamma=round(10 ** rng.uniform(-4, -2), 7), iters=rng.randint(8, 24))
    if kind == "train":
        return dict(kind=kind, n=rng.choice([64, 96, 128]), samples=rng.choice([64, 128, 192]), batch=rng.choice([16, 32]))
    if kind == "dirk":
        return dict(kind=kind, nx=_log(rng, 32, 128), ny=_log(rng, 32, 128), order=rng.choice([2, 3]),
                    ls=rng.choice(["cg", "gmres"]), prec=rng.choice(["jacobi", "pfmg"]),
                    tf=round(rng.uniform(0.02, 0.1), 3))
    return dict(kind=kind, n=_log(rng, 1000, 3e7))


# ---------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator()
    g.manual_seed(seed)
    return g


def _grid(n):
    return (torch.arange(n, dtype=torch.float64, device="cuda") + 1.0) / (n + 1)


def _modes(nx, ny, seed, count=8, pmax=16):
    """A seeded sum of sine modes on the interior grid (ny x nx), of unit size."""
    g = _gen(seed)
    p = torch.randint(1, pmax + 1, (count,), generator=g).double().cuda()
    q = torch.randint(1, pmax + 1, (count,), generator=g).double().cuda()
    a = torch.randn(count, generator=g, dtype=torch.float64).cuda() / math.sqrt(count)
    sx = torch.sin(math.pi * p[:, None] * _grid(nx)[None, :])
    sy = torch.sin(math.pi * q[:, None] * _grid(ny)[None, :]) * a[:, None]
    return sy.t() @ sx


def _bumps(nx, ny, seed, count=24):
    """A seeded smooth right-hand side: Gaussian bumps."""
    g = _gen(seed)
    cx, cy = (0.1 + 0.8 * torch.rand(count, generator=g, dtype=torch.float64) for _ in range(2))
    w = 0.03 + 0.12 * torch.rand(count, generator=g, dtype=torch.float64)
    a = torch.randn(count, generator=g, dtype=torch.float64)
    cx, cy, w, a = (v.cuda() for v in (cx, cy, w, a))
    ex = torch.exp(-(_grid(nx)[None, :] - cx[:, None]) ** 2 / (2 * w[:, None] ** 2))
    ey = torch.exp(-(_grid(ny)[None, :] - cy[:, None]) ** 2 / (2 * w[:, None] ** 2)) * a[:, None]
    return ey.t() @ ex


def _start(c, seed):
    """The manufactured initial state with a seeded perturbation (forced), or seeded modes."""
    m = _modes(c["nx"], c["ny"], seed)
    if not c.get("forced", True):
        return m
    s = torch.sin(math.pi * _grid(c["ny"])) ** 2
    return torch.outer(s, torch.sin(math.pi * _grid(c["nx"])) ** 2) + 0.05 * m


def _periodic_start(c, seed):
    """The reference's initial state (Gaussian in y, sine in x) with a seeded perturbation."""
    g = _gen(seed)
    a = torch.randn(4, generator=g, dtype=torch.float64)
    x = -math.pi + 2 * math.pi * torch.arange(c["nx"], dtype=torch.float64, device="cuda") / (c["nx"] - 1)
    y = -6.0 + 12.0 * torch.arange(c["ny"], dtype=torch.float64, device="cuda") / (c["ny"] - 1)
    fx = 1.0 + 0.3 * torch.sin(2 * x)
    for k in range(4):
        fx = fx + 0.05 * float(a[k]) * torch.sin((k + 1) * x)
    return torch.outer(torch.exp(-y * y / 5.5) / math.sqrt(5.5 * math.pi), fx)


def _vectors(n, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return [torch.randn(n, generator=g, dtype=torch.float64, device="cuda") for _ in range(5)]


def _bound(c):
    """A bound of the operator's spectral radius, as a user's dom_eig function gives it."""
    if c["kind"] == "sts":
        return 4.0 * (c["kx"] * (c["nx"] + 1.0) ** 2 + c["ky"] * (c["ny"] + 1.0) ** 2)
    most = 1.99 if c["inhom"] else 1.0  # k (1 + 0.99 sin)
    return 4.0 * most * (c["kx"] * ((c["nx"] - 1) / (2 * math.pi)) ** 2 + c["ky"] * ((c["ny"] - 1) / 12.0) ** 2)


def _h_rho(method, s):
    """h rho for which the integrator takes s stages."""
    if method == "rkc":
        return ((s - 0.5) ** 2 - 1.0) / 1.54
    return 0.999 * ((2 * s + 1) ** 2 - 9.0) / 8.0


def _method(c):
    return sts.RKC if c["method"] == "rkc" else sts.RKL


def _batch_sizes(c):
    return [int(n) for n in np.random.default_rng(c["count"]).choice((64, 96, 128, 192, 256, 384, 512), c["count"])]


def _batch_instances(c, seed):
    rng = np.random.default_rng(seed)
    inst, state = [], []
    for n in _batch_sizes(c):
        kx, ky = (float(10 ** rng.uniform(-2, 0)) for _ in range(2))
        p, q = rng.integers(1, 17, 8), rng.integers(1, 17, 8)
        a = rng.standard_normal(8)
        x = (np.arange(n) + 1.0) / (n + 1)
        state.append(((np.sin(np.pi * np.outer(q, x)) * a[:, None]).T @ np.sin(np.pi * np.outer(p, x))).ravel())
        inst.append((n, kx, ky, np.array([1]), np.array([1]), np.array([0.0])))
    return inst, np.concatenate(state)


def prepare(case, seed):
    c, ctx = case, _context()
    kind = c["kind"]
    s = dict(case=c, kind=kind, ctx=ctx)
    if kind in ("solve", "sts"):
        s["problem"] = sts.Problem(ctx, sts.MANUFACTURED if c.get("forced", True) else sts.UNFORCED, c["nx"], c["ny"],
                                   c["kx"], c["ky"])
        s["y0"] = _start(c, seed).contiguous()
    if kind == "refmode":
        s["problem"] = sts.Problem(ctx, sts.PERIODIC, c["nx"], c["ny"], c["kx"], c["ky"], inhomogeneous=c["inhom"])
        s["y0"] = _periodic_start(c, seed).contiguous()
    if kind == "dirk":
        s["problem"] = sts.Problem(ctx, sts.PERIODIC, c["nx"], c["ny"], 1.0, 0.5, inhomogeneous=True)
        s["y0"] = _periodic_start(c, seed).contiguous()
    if "y0" in s:
        s["y"] = torch.empty_like(s["y0"])
        s["v0"], s["v"] = _wrap(ctx, s["y0"]), _wrap(ctx, s["y"])
    if kind in ("sts", "refmode"):
        # the step size that needs the case's stage count; the integrator is kept between runs
        bound = _bound(c)
        s["h"] = _h_rho(c["method"], c["stages"]) / (1.01 * bound)
        torch.cuda.synchronize()
        s["integrator"] = sts.LSRKStep(ctx, s["problem"], 0.0, s["v0"], method=_method(c), rtol=1e-6, atol=1e-10,
                                       mixed=c["mixed"], hfixed=s["h"], dom_eig=lambda t: -bound)
    if kind == "dirk" and c["prec"] == "pfmg":
        s["mg"] = sts.PFMG(s["problem"])
    if kind == "batch":
        inst, s["state"] = _batch_instances(c, seed)
        s["batch"] = sts.Batch(ctx, inst)
        s["batch"].set_mixed(c["mixed"])
        s["batch"].set_launch(256, 4, 8, 256)
    if kind in ("pcg", "pfmg", "learned"):
        nx, ny = (c["n"], c["n"]) if kind == "learned" else (c["nx"], c["ny"])
        s["problem"] = sts.Problem(ctx, sts.UNFORCED, nx, ny, 1.0, c["ky"])
        s["b"] = _bumps(nx, ny, seed).contiguous()
        s["x"] = torch.empty_like(s["b"])
        s["vb"], s["vx"] = _wrap(ctx, s["b"]), _wrap(ctx, s["x"])
        if kind == "learned":
            s["net"] = sts.Net(ctx, nx, seed=seed % 1000)
    if kind == "train":
        s.update(_training_set(c, seed))
        s["net"] = sts.Net(ctx, c["n"], seed=seed % 1000)
    if kind == "nvector":
        s["t"] = _vectors(c["n"], seed)
        s["out"] = [torch.empty_like(s["t"][0]) for _ in range(2)]
        s["x"] = [_wrap(ctx, t) for t in s["t"]]
        s["z"], s["w"] = (_wrap(ctx, t) for t in s["out"])
    torch.cuda.synchronize()
    return s


def _training_set(c, seed):
    """Residual / correction pairs r = (I - gamma A) e of smooth corrections, with metadata."""
    n, count = c["n"], c["samples"]
    rng = np.random.default_rng(seed)
    dx = 1.0 / (2048 + 1)
    r = torch.empty(count, n, n, device="cuda")
    e = torch.empty(count, n, n, device="cuda")
    meta = np.empty((count, 7), dtype=np.float32)
    for k in range(count):
        ky, gamma = 10 ** rng.uniform(-3, 0), 10 ** rng.uniform(-4, -2)
        sk, sg, jac, gcx, gcy = sts.net_features(1.0, ky, gamma, dx)
        ek = _modes(n, n, int(rng.integers(1 << 31)), count=12, pmax=24)
        pad = torch.nn.functional.pad(ek, (1, 1, 1, 1))
        rk = ek - gcx * (pad[1:-1, :-2] - 2 * ek + pad[1:-1, 2:]) - gcy * (pad[:-2, 1:-1] - 2 * ek + pad[2:, 1:-1])
        norm, energy = torch.stack([rk.square().mean().sqrt(), (ek * rk).sum()]).tolist()
        r[k], e[k] = rk, ek
        meta[k] = (sk, sg, jac, 1.0 / norm, 1.0 / energy, gcx, gcy)
    return dict(r=r, e=e, meta=torch.from_numpy(meta).cuda())


# ---------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------
def run(state):
    s, c, kind = state, state["case"], state["kind"]
    if kind == "solve":
        I = sts.LSRKStep(s["ctx"], s["problem"], 0.0, s["v0"], method=_method(c), rtol=1e-6, atol=1e-10,
                         mixed=c["mixed"])
        I.set_stop_time(c["tf"])
        I.evolve(c["tf"], s["v"])
        steps = I.stats()["nst"]
        I.free()
        return dict(y=s["y"], steps=steps)
    if kind in ("sts", "refmode"):
        I, tf = s["integrator"], c["steps"] * s["h"]
        I.reset(0.0, s["v0"])
        I.set_stop_time(tf)
        I.evolve(tf, s["v"])
        return s["y"]
    if kind == "dirk":
        I = sts.ARKStep(s["ctx"], s["problem"], 0.0, s["v0"], implicit=True, order=c["order"], rtol=1e-5, atol=1e-10,
                        controller=sts.I, ls=c["ls"], prec=c["prec"], pfmg=s.get("mg"))
        I.set_stop_time(c["tf"])
        I.evolve(c["tf"], s["v"])
        iters = I.stats()["nli"]
        I.free()
        return dict(y=s["y"], iters=iters)
    if kind == "batch":
        B = s["batch"]
        B.set_state(s["state"])
        B.evolve(c["tf"], method=sts.RKL, rtol=1e-6, atol=1e-10)
        return B.state()
    if kind == "pcg":
        iters, res, _ = sts.implicit_solve_pcg(s["problem"], c["gamma"], s["vb"], s["vx"], tol=1e-8)
        return dict(x=s["x"], iters=iters)
    if kind == "pfmg":
        mg = sts.PFMG(s["problem"], relax=c["relax"])
        iters, res, _ = sts.implicit_solve_pfmg(s["problem"], c["gamma"], mg, s["vb"], s["vx"], tol=1e-8)
        return dict(x=s["x"], iters=iters)
    if kind == "learned":
        # a fixed number of iterations (a tolerance that is not reached, no fallback)
        sts.fcg_solve(s["problem"], c["gamma"], s["net"], s["vb"], s["vx"], tol=1e-14, maxit=-c["iters"])
        return s["x"]
    if kind == "train":
        loss = s["net"].train(c["n"], c["samples"], s["r"].data_ptr(), s["e"].data_ptr(), s["meta"].data_ptr(), 1,
                              c["batch"], 1e-3, seed=3)
        return dict(loss=loss, weights=s["net"].weights())
    # one step's vector work: a stage combination, the error weight and its norm, a dot product
    x, z, w = s["x"], s["z"], s["w"]
    z.linear_combination([0.7, -0.2, 0.5, 1e-3, -2e-3], x)
    w.abs(x[0])
    w.scale(1e-4, w)
    w.add_const(w, 1e-2)
    w.inv(w)
    norm = z.wrms_norm(w)
    dot = z.dot(x[1])
    top = z.max_norm()
    return dict(z=s["out"][0], w=s["out"][1], norm=norm, dot=dot, top=top)


# ---------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------
def work(case):
    c, kind = case, case["kind"]
    if kind == "solve":
        n = c["nx"] * c["ny"]
        rho = 8.0 * max(c["kx"] * c["nx"] ** 2, c["ky"] * c["ny"] ** 2)
        steps = 1500.0 * c["tf"]  # about what rtol 1e-6 takes
        stages = math.sqrt(rho * c["tf"] / steps) + 1
        return dict(bytes=16.0 * n, flops=17.0 * n * stages * steps)
    if kind in ("sts", "refmode"):
        # state in and out once per step with its derivative; the recurrence per stage
        n = c["nx"] * c["ny"]
        return dict(bytes=32.0 * n * c["steps"], flops=17.0 * n * c["stages"] * c["steps"])
    if kind == "batch":
        n = sum(k * k for k in _batch_sizes(c))
        return dict(bytes=16.0 * n, flops=17.0 * n * 4e5 * c["tf"])  # about 4e5 stages per unit of time
    if kind in ("pcg", "pfmg"):
        n = c["nx"] * c["ny"]
        if kind == "pfmg":
            return dict(bytes=16.0 * n, flops=80.0 * n * 10)
        kappa = 1.0 + 4.0 * c["gamma"] * ((c["nx"] + 1) ** 2 + c["ky"] * (c["ny"] + 1) ** 2)
        return dict(bytes=16.0 * n, flops=17.0 * n * 9.0 * math.sqrt(kappa))
    if kind == "learned":
        n = c["n"] ** 2
        return dict(bytes=16.0 * n, flops=(20.0 + 300.0 + 2 * 2304.0 * 0.33 * 2) * n * c["iters"])
    if kind == "train":
        n = c["n"] ** 2 * c["samples"]
        return dict(bytes=8.0 * n, flops=3.0 * 2.0 * (2 * 432 + 2 * 2304 * 0.33) * n)
    if kind == "dirk":
        n = c["nx"] * c["ny"]
        return dict(bytes=16.0 * n, flops=20.0 * n * 1000 * c["tf"])
    return dict(bytes=8.0 * c["n"] * 7, flops=20.0 * c["n"])


# ---------------------------------------------------------------------------------------
# the same in plain 64-bit arithmetic
# ---------------------------------------------------------------------------------------
def _coeffs(method, s):
    """mu, nu, mus, a_{j-1}, c_{j-1} of the RKC2 / RKL2 recurrences, j = 1 .. s."""
    mu, nu, mus, a, cj = ([0.0] * (s + 1) for _ in range(5))
    if method == "rkl":
        w1 = 4.0 / ((s + 2.0) * (s - 1.0))
        b = [1.0 / 3.0] * 3 + [(j * j + j - 2.0) / (2.0 * j * (j + 1.0)) for j in range(3, s + 1)]
        mus[1] = w1 * b[1]
        cs = [0.0, w1 * b[1]] + [(j * j + j - 2.0) * w1 / 4.0 for j in range(2, s + 1)]
        for j in range(2, s + 1):
            mu[j] = (2 * j - 1.0) / j * b[j] / b[j - 1]
            nu[j] = -(j - 1.0) / j * b[j] / b[j - 2]
            mus[j], a[j], cj[j] = mu[j] * w1, 1.0 - b[j - 1], cs[j - 1]
        return mu, nu, mus, a, cj
    w0 = 1.0 + 2.0 / (13.0 * s * s)
    T, dT, d2T = [1.0, w0], [0.0, 1.0], [0.0, 0.0]
    for j in range(2, s + 1):
        T.append(2 * w0 * T[-1] - T[-2])
        dT.append(2 * w0 * dT[-1] - dT[-2] + 2 * T[j - 1])
        d2T.append(2 * w0 * d2T[-1] - d2T[-2] + 4 * dT[j - 1])
    w1 = dT[s] / d2T[s]
    b = [0.0, 0.0] + [d2T[j] / dT[j] ** 2 for j in range(2, s + 1)]
    b[0] = b[1] = 1.0 / (4.0 * w0 * w0)
    mus[1] = w1 * b[1]
    th = [0.0, mus[1]]
    for j in range(2, s + 1):
        mu[j], nu[j] = 2 * w0 * b[j] / b[j - 1], -b[j] / b[j - 2]
        mus[j], a[j], cj[j] = 2 * w1 * b[j] / b[j - 1], 1.0 - T[j - 1] * b[j - 1], th[j - 1]
        th.append(mu[j] * th[j - 1] + nu[j] * th[j - 2] + mus[j] * (1.0 - a[j]))
    return mu, nu, mus, a, cj


def _rhs_dirichlet(c):
    nx, ny = c["nx"], c["ny"]
    cx, cy = c["kx"] * (nx + 1.0) ** 2, c["ky"] * (ny + 1.0) ** 2
    px, py = math.pi * _grid(nx), math.pi * _grid(ny)
    Sx, Sy = torch.sin(px) ** 2, torch.sin(py) ** 2
    Dx, Dy = 2 * math.pi ** 2 * torch.cos(2 * px), 2 * math.pi ** 2 * torch.cos(2 * py)

    def f(t, u):
        out = u * (-2.0 * (cx + cy))
        out[:, 1:] += cx * u[:, :-1]
        out[:, :-1] += cx * u[:, 1:]
        out[1:] += cy * u[:-1]
        out[:-1] += cy * u[1:]
        if c["forced"]:  # b = u*_t - kx u*_xx - ky u*_yy for u* = S(x) S(y) cos^2(2 pi t)
            q = math.cos(2 * math.pi * t) ** 2
            qt = -2 * math.pi * math.sin(4 * math.pi * t)
            out.addr_(Sy, qt * Sx - c["kx"] * q * Dx)
            out.addr_(Dy, Sx, alpha=-c["ky"] * q)
        return out

    return f


def _rhs_periodic(c):
    nx, ny = c["nx"], c["ny"]
    dx, dy = 2 * math.pi / (nx - 1), 12.0 / (ny - 1)
    i = torch.arange(nx, dtype=torch.float64, device="cuda")
    j = torch.arange(ny, dtype=torch.float64, device="cuda")

    def k(v, x):
        return v * (1.0 + 0.99 * torch.sin(x)) if c["inhom"] else v + 0.0 * x

    w, e = (k(c["kx"], -math.pi + (i + o) * dx) / dx ** 2 for o in (-0.5, 0.5))
    s, n = (k(c["ky"], -6.0 + (j + o) * dy)[:, None] / dy ** 2 for o in (-0.5, 0.5))

    def f(t, u):
        return (w * (torch.roll(u, 1, 1) - u) + e * (torch.roll(u, -1, 1) - u) + s * (torch.roll(u, 1, 0) - u)
                + n * (torch.roll(u, -1, 0) - u))

    return f


def _steps(c, f, y, h):
    mu, nu, mus, a, cj = _coeffs(c["method"], c["stages"])
    t, tf = 0.0, c["steps"] * h
    for k in range(c["steps"]):
        if k == c["steps"] - 1:
            h = tf - t  # the stop time ends the last step
        f0 = f(t, y)
        d2, d1 = torch.zeros_like(y), (h * mus[1]) * f0  # increments from the step's start
        for j in range(2, c["stages"] + 1):
            d = f(t + h * cj[j], y + d1)
            d.sub_(f0, alpha=a[j]).mul_(h * mus[j]).add_(d1, alpha=mu[j]).add_(d2, alpha=nu[j])
            d2, d1 = d1, d
        y = y + d1
        t += h
    return y


def _shifted_solve(c, b):
    """(I - gamma A)^-1 b by sine transforms (the eigenvectors of the Dirichlet operator)."""
    ny, nx = b.shape
    lx, ly = (4.0 * k * (n + 1.0) ** 2 * torch.sin(0.5 * math.pi * _grid(n)) ** 2
              for k, n in ((1.0, nx), (c["ky"], ny)))

    def dst(u):  # DST-I along the last axis, unnormalised
        n = u.shape[-1]
        z = torch.zeros(u.shape[:-1] + (1,), dtype=u.dtype, device=u.device)
        return -torch.fft.rfft(torch.cat([z, u, z, -u.flip(-1)], -1))[..., 1:n + 1].imag.contiguous()

    v = dst(dst(b).t().contiguous()).t()
    v = (v / (1.0 + c["gamma"] * (ly[:, None] + lx[None, :]))).contiguous()
    v = dst(dst(v).t().contiguous()).t()
    return v / (4.0 * (nx + 1.0) * (ny + 1.0))


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "sts":
        return _steps(c, _rhs_dirichlet(c), _start(c, seed), _h_rho(c["method"], c["stages"]) / (1.01 * _bound(c)))
    if kind == "refmode":
        return _steps(c, _rhs_periodic(c), _periodic_start(c, seed),
                      _h_rho(c["method"], c["stages"]) / (1.01 * _bound(c)))
    if kind in ("pcg", "pfmg"):
        return dict(x=_shifted_solve(c, _bumps(c["nx"], c["ny"], seed)), iters=None)
    if kind == "nvector":
        x = _vectors(c["n"], seed)
        z = 0.7 * x[0] - 0.2 * x[1] + 0.5 * x[2] + 1e-3 * x[3] - 2e-3 * x[4]
        w = 1.0 / (1e-4 * x[0].abs() + 1e-2)
        return dict(z=z, w=w, norm=float((z * w).square().mean().sqrt()), dot=float((z * x[1]).sum()),
                    top=float(z.abs().max()))
    return None  # adaptive integrations, 16-bit networks: no closed 64-bit form of the same outputs

