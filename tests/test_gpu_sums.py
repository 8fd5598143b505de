"""Sums of products and of pair groups against plain torch float64 transforms, with
bounds that the library's own sums have no part in.

Tolerances:
  * PS_FP64_PLAIN  : |dB| <= 1e-9 |B| + n 1e-15 A
  * PS_FP32_BATCHED: |dB| <= 1e-5 |B| + n 3e-7 A
A the reference's sum of the terms' absolute values in the units of B: a leg carries
about 3e-7 of its size in FP32 (2^-24 per rounding, some 10 roundings in each of three
passes, random signs), the n legs' errors adding up; 1e-15 in FP64 likewise.  Counts
are equal after rounding, in PS_FP32_BATCHED as they are.
"""
import numpy as np
import pytest

from polyspectrum_b200 import synth

pytestmark = pytest.mark.gpu

BOX = 150.0
KF = 2 * np.pi / BOX


def by_torch(field, cfgs):
    """B, A and counts of DEFAULT and GIVEN configurations."""
    import torch
    n = field.shape[0]
    L = float(np.float32(BOX))
    kf = 2 * np.pi / L
    dk = torch.fft.rfftn(field)
    m = torch.fft.fftfreq(n, 1.0 / n, dtype=torch.float64, device=field.device)
    mz = torch.arange(n // 2 + 1, dtype=torch.float64, device=field.device)
    r = torch.sqrt(m[:, None, None] ** 2 + m[None, :, None] ** 2 + mz[None, None, :] ** 2)
    out = []
    for g in cfgs:
        d = i = None
        half = 0.5 * g.kbinwidth
        for l in range(g.n):
            if g.kbinningCase == 2 and l == g.n - 1:
                mask = (g.kmin[l] / kf - r <= half) & (r - g.kmax[l] / kf <= half)
            else:
                mask = (g.k[l] / kf - r).abs() <= half
            x = torch.fft.irfftn(dk * mask, s=field.shape, norm="forward")
            d = x if d is None else d.mul_(x)
            x = torch.fft.irfftn(mask.to(dk.dtype), s=field.shape, norm="forward")
            i = x if i is None else i.mul_(x)
            del x, mask
        si = float(i.sum())
        np_ = np.rint(si / float(n) ** 3)
        coef = L ** (3 * (g.n - 1)) / float(n) ** (3 * g.n) / (np_ * float(n) ** 3) if np_ else np.nan
        out.append((coef * float(d.sum()), abs(coef) * float(d.abs().sum()), np_))
    return np.array(out).T


def check(ps, n_grid, field, cfgs, ref, singly=True):
    rB, A, rN = ref
    has = rN > 0
    assert has.any()
    legs = np.array([g.n for g in cfgs])
    for method, rel, eps in ((1, 1e-9, 1e-15), (2, 1e-5, 3e-7)):
        bound = rel * np.abs(rB) + eps * legs * A

        def compare(B, Np, s=slice(None)):
            np.testing.assert_array_equal(Np if method == 2 else np.rint(Np), rN[s])
            err = np.abs(B - rB[s])
            assert np.all((err <= bound[s])[has[s]]), (err / bound[s])[has[s]]

        with ps.Context(n_grid, BOX, methods=method) as ctx:
            ctx.get_FT_field(ps.PS_FIELD_DENS, field)
            B, Np, _, _ = ctx.batch(cfgs, method)
            compare(B, Np)
            Bk, Nk, kap, _ = ctx.batch(cfgs, method, kappa=True)  # the same sums beside the absolute ones
            np.testing.assert_array_equal(Nk, Np)
            np.testing.assert_array_equal(Bk, B)
            three = has & (legs > 2)
            assert np.isfinite(kap[three]).all() and (kap[three] >= 1 - 1e-6).all()
            if singly:
                for q in range(len(cfgs)):
                    B1, N1, _, _ = ctx.batch(cfgs[q:q + 1], method)
                    compare(B1, N1, slice(q, q + 1))


@pytest.mark.parametrize("n_grid", [16, 48, 60])
@pytest.mark.parametrize("kb", [0, 2])
def test_products(gpu_lib, n_grid, kb):
    """n = 3 to 8: powers of one leg, several distinct legs, sub-grids and the whole grid."""
    import torch
    ps = gpu_lib
    top = 0.45 * n_grid
    rng = np.random.default_rng(10 * n_grid + kb)
    sets = [[a] * 4 for a in rng.uniform(1.6, top, 3)]
    sets += [[a, a, b, b] for a, b in rng.uniform(1.6, 4.0, (3, 2))]
    sets += [list(v) for v in rng.uniform(1.6, 3.4, (20, 4))] + [list(v) for v in rng.uniform(1.6, top, (3, 4))]
    sets += [[a, a, a, b, a] for a, b in rng.uniform(1.6, 3.4, (3, 2))] + [[1.7, 2.2, 2.6] * 2] + [[1.2] * 7, [1.2] * 8]
    sets += [list(v) for v in rng.uniform(1.6, 0.6 * top, (6, 3))]
    cfgs = [ps.make_cfg(len(s), [k * KF for k in s], [0.0] * (len(s) - 1) + [(s[-1] - 0.6) * KF],
                        [0.0] * (len(s) - 1) + [(s[-1] + 0.8) * KF], 1.0, kb) for s in sets]
    field = synth.lognormal_density(n_grid, 2.0, 6).astype(np.float32)
    check(ps, n_grid, field, cfgs, by_torch(torch.from_numpy(field).cuda().double(), cfgs))


@pytest.mark.parametrize("n_grid,top", [(96, 20.0), (128, 60.0), (192, 62.0), (256, 90.0), (300, 60.0), (320, 150.0),
                                        (384, 120.0), (512, 90.0), (600, 125.0)])
def test_lengths(gpu_lib, n_grid, top):
    import torch
    ps = gpu_lib
    torch.manual_seed(n_grid)
    field = torch.randn((n_grid,) * 3, device="cuda", dtype=torch.float32).exp_()
    top += 0.137  # no mode on an edge of a shell
    sides = [[top, 0.67 * top, 0.51 * top], [0.67 * top, 0.67 * top, top], [0.8 * top] * 3, [0.12 * top] * 4, [top] * 2]
    cfgs = [ps.make_cfg(len(s), [k * KF for k in s], kbinwidth=3.0) for s in sides]
    ref = by_torch(field.double(), cfgs)
    torch.cuda.empty_cache()
    check(ps, n_grid, field, cfgs, ref, singly=False)


def test_legs_one_by_one(gpu_lib):
    """1024 points, four full-grid FP64 legs (above the memory of a product's spectra)."""
    import torch
    ps = gpu_lib
    torch.manual_seed(3)
    field = torch.randn((1024,) * 3, device="cuda", dtype=torch.float32).exp_()
    cfgs = [ps.make_cfg(4, [k * KF for k in (300.137, 310.21, 320.33, 200.41)], kbinwidth=0.1)]
    ref = by_torch(field.double(), cfgs)
    torch.cuda.empty_cache()
    check(ps, 1024, field, cfgs, ref, singly=False)
