"""Polygon counts by FP64 transforms of the unit shells (PS_PLAN_FFT_COUNTS) against
the enumeration in integers: whole numbers, equal."""
import numpy as np
import pytest

from polyspectrum_b200 import synth

pytestmark = pytest.mark.gpu

BOX = 150.0


# sides of 0.34 N modes keep the transforms on the N-grid, whose (N/2 + 1)^2 rows of the
# quadrant end in a tile that is only partly filled, with idle and busy rows in one warp
# for rows of fewer than 32 threads
@pytest.mark.parametrize("n_grid", [16, 32, 48, 60, 64, 96, 128, 192, 256, 300, 320, 384])
@pytest.mark.parametrize("two", [False, True])
def test_partly_filled_row_tiles(gpu_lib, n_grid, two):
    ps = gpu_lib
    kf = 2 * np.pi / BOX
    a = 0.34 * n_grid + 0.137
    sides = [(a, a + 1.3 * two, c) for c in (a, 0.9 * a, 0.5 * a)]
    cfgs = [ps.make_cfg(3, [k * kf for k in s], kbinwidth=0.9) for s in sides]
    field = synth.lognormal_density(n_grid, 2.0, 3)
    with ps.Context(n_grid, BOX, methods=ps.PS_FP32_BATCHED) as ctx:
        ctx.get_FT_field(ps.PS_FIELD_DENS, field)
        got = []
        for fft in (False, True):
            p = ctx.plan(cfgs, fft_counts=fft)
            got.append(p.execute()[1])
            p.close()
    assert (got[0] > 0).all()
    np.testing.assert_array_equal(got[1], got[0])
