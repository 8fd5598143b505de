"""Field loads limited to a plan's band (ps_gpu_set_spectrum_band) at the lengths whose
field passes have geometries of their own: the plan's results are those of a full load,
bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BOX = 150.0
KF = 2 * np.pi / BOX


@pytest.mark.parametrize("n_grid,top", [(256, 40.0), (512, 70.0), (1024, 60.0), (1024, 200.0)])
@pytest.mark.parametrize("phase", [0, 1])
def test_band_limited_load(gpu_lib, n_grid, top, phase):
    import torch
    ps = gpu_lib
    torch.manual_seed(n_grid)
    field = torch.randn((n_grid,) * 3, device="cuda", dtype=torch.float32).exp_()
    cfgs = [ps.make_cfg(2, [k * KF, k * KF]) for k in np.linspace(1.5, top, 40)]
    cfgs += [ps.make_cfg(3, [a * KF, a * KF, 0.7 * a * KF], kbinwidth=0.5) for a in (0.3 * top, 0.4 * top)]
    with ps.Context(n_grid, BOX, methods=ps.PS_FP32_BATCHED) as ctx:
        plan = ctx.plan(cfgs)
        got = []
        for band in (-1, plan.band):
            ctx.set_spectrum_band(band)
            ctx.get_FT_field(ps.PS_FIELD_DENS, field, use_only_phase=phase)
            got.append(plan.execute()[:2])
        assert plan.band < n_grid // 2
        plan.close()
    assert np.isfinite(got[0][0]).all() and (got[0][1] > 0).all()
    np.testing.assert_array_equal(got[1][1], got[0][1])
    np.testing.assert_array_equal(got[1][0], got[0][0])
