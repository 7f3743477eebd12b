"""A solve that has returned is complete: its result may be read on any stream."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("solver", ["PCGSolver", "SPGMRSolver", "SPFGMRSolver"])
def test_result_of_a_generic_solve_on_another_stream(ctx, stslib, solver):
    n, gamma = 2048, 1e-3
    P = stslib.Problem(ctx, 1, n, n, 1.0, 0.1)
    torch.manual_seed(3)
    b, x = torch.randn(n * n, dtype=torch.float64, device="cuda"), torch.zeros(n * n, dtype=torch.float64, device="cuda")
    vb, vx = (stslib.NVector(ctx, handle=stslib.lib().N_VMake_Sts(t.numel(), t.data_ptr(), ctx.h)) for t in (b, x))
    S = getattr(stslib, solver)(ctx, vb, maxl=24, precond=True)
    other = torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(5):
        stslib.implicit_solve_ls(P, gamma, S, vb, vx, tol=1e-14)  # (ends unconverged after 24 iterations)
        with torch.cuda.stream(other):
            seen = x.clone()
        torch.cuda.synchronize()
        assert torch.equal(seen, x)
        x.zero_()
        torch.cuda.synchronize()
