"""The times that the stage kernel's getters report are of the choice in use: 0 where that was taken
untimed, whatever an earlier setting had timed."""
import pytest

pytestmark = pytest.mark.gpu


def test_times_of_an_earlier_setting_are_dropped(ctx, stslib):
    P = stslib.Problem(ctx, 0, 300, 200, 1.0, 0.3)
    I = stslib.LSRKStep(ctx, P, 0.0, P.initial(), mixed=True, hfixed=1e-4, stage_fusion=(1, 0))
    y = P.vector()
    t = 1e-3
    for ks, timed in ((1, True), (0, False), (4, True), (0, False)):
        assert stslib.lib().STS_LSRKStepSetStageFusion(I.mem, ks, 0) == 0
        I.evolve(t, y)
        t += 1e-3
        info, group = I.stage_kernel_info(), I.stage_fusion_info()
        assert (info["ms"] > 0.0) == timed
        assert group["ks"] == (ks or 8) and (group["ms"] > 0.0) == (ks == 4)
