"""Batched launches, shell lists, packed real transforms and two-pass transform
lengths at the sizes where their tiling and dispatch change.

Small grids are compared with the CPU oracle, larger ones with a plain torch
float64 transform of the same estimator (masked spectra, inverse real
transforms, sums of products).

Tolerances, fixed by the methods' arithmetic:
  * PS_FP64_PLAIN  : |dB| <= 1e-9 |B| + 1e-11 max|B|; counts equal after rounding
  * PS_FP32_BATCHED: |dB| <= 1e-5 |B| + 1e-6 max|B|; counts exactly equal
    (2^-24 per rounding, some 10 roundings per transform pass, random signs)
  * gradients: FP64 1e-9 max|g|, FP32 1e-4 max|g|
  * where the terms of single sums cancel: |dB| <= (10 eps) kappa |B| on top, with
    kappa = sum |terms| / |sum terms| and eps = 1e-16 / 1e-7
B of a configuration without polygons is 0/0 and not compared.
"""
import threading

import numpy as np
import pytest

from polyspectrum_b200 import synth

pytestmark = pytest.mark.gpu

TOL = {1: (1e-9, 1e-11), 2: (1e-5, 1e-6)}
BOX = 150.0


def check(method, B, Np, rB, rN, kappa=None):
    rt, at = TOL[method]
    rN = np.rint(rN)
    has = rN != 0
    np.testing.assert_array_equal(np.rint(Np), rN)
    if method == 2:
        np.testing.assert_array_equal(Np, rN)
    if has.any():
        scale = np.abs(rB[has]).max()
        err = np.abs(B - rB)[has]
        bound = rt * np.abs(rB[has]) + at * scale
        if kappa is not None:
            bound += {1: 1e-15, 2: 1e-6}[method] * kappa[has] * np.abs(rB[has])
        assert np.all(err <= bound), (err / np.abs(rB[has]), err / bound)


def by_oracle(ora, n_grid, field, cfgs, phase=0):
    L = float(np.float32(BOX))
    dk = ora.ora_forward(n_grid, 0, field, None, phase)
    B, Np = np.zeros(len(cfgs)), np.zeros(len(cfgs))
    for q, g in enumerate(cfgs):
        k, lo, hi = ([a[i] for i in range(g.n)] for a in (g.k, g.kmin, g.kmax))
        B[q], _, _, lo, hi = ora.ora_polyspectrum(n_grid, dk, k, lo, hi, g.kbinwidth, g.kbinningCase, L)
        Np[q] = ora.ora_num_polygons(n_grid, k, lo, hi, g.kbinwidth, g.kbinningCase, L)
    return B, Np


def by_torch(field, cfgs, phase=False):
    """The estimator with torch float64 transforms (DEFAULT shells); field may
    require a gradient (then B stay tensors)."""
    import torch
    n = field.shape[0]
    L = float(np.float32(BOX))
    kf = 2 * np.pi / L
    dk = torch.fft.rfftn(field)
    if phase:
        a = dk.abs()
        dk = dk / torch.where(a > 0, a, 1.0)
    m = torch.fft.fftfreq(n, 1.0 / n, dtype=torch.float64, device=field.device)
    mz = torch.arange(n // 2 + 1, dtype=torch.float64, device=field.device)
    r = torch.sqrt(m[:, None, None] ** 2 + m[None, :, None] ** 2 + mz[None, None, :] ** 2)
    Bs, Ns = [], []
    for g in cfgs:
        d = i = 1.0
        for l in range(g.n):
            mask = ((r * kf - g.k[l]).abs() <= 0.5 * g.kbinwidth * kf).to(torch.float64)
            d = d * torch.fft.irfftn(dk * mask, s=field.shape, norm="forward")
            i = i * torch.fft.irfftn(mask + 0j, s=field.shape, norm="forward")
        si = i.sum()
        Bs.append(L ** (3 * (g.n - 1)) / float(n) ** (3 * g.n) * d.sum() / si)
        Ns.append(float(si) / float(n) ** 3)
    return Bs, np.array(Ns)


def triangles(ps, n_grid, count, top, kb, seed, bw=1.0):
    """Random closing triangles of sides up to `top` modes."""
    kf = 2 * np.pi / BOX
    rng = np.random.default_rng(seed)
    cfgs = []
    while len(cfgs) < count:
        a, b = rng.uniform(1.6, top, 2)
        c = np.sqrt(max(a * a + b * b + 2 * a * b * rng.uniform(-0.9, 0.9), 0.0))
        if not 1.6 < c < top:
            continue
        cfgs.append(ps.make_cfg(3, [a * kf, b * kf, c * kf], [0.0, 0.0, (c - 0.4) * kf],
                                [0.0, 0.0, (c + 0.7) * kf], bw, kb))
    return cfgs


@pytest.mark.parametrize("n_grid", [16, 48, 60])
@pytest.mark.parametrize("kb", [0, 2, 3])
@pytest.mark.parametrize("bw", [0.3, 1.0, 3.0])
def test_shell_lists(gpu_lib, ora, n_grid, kb, bw):
    """n = 2: overlapping, repeated, unordered and empty shells, to the corner modes."""
    ps = gpu_lib
    kf = 2 * np.pi / BOX
    rng = np.random.default_rng(n_grid)
    ks = np.concatenate([rng.uniform(0.6, 0.9 * n_grid, 24), [2.2, 2.2, 3.0 * n_grid]])
    cfgs = [ps.make_cfg(2, [k * kf, k * kf], [0.0, (k - 0.2) * kf], [0.0, (k + 0.9) * kf], bw, kb) for k in ks]
    field = synth.lognormal_density(n_grid, 2.0, 4)
    rB, rN = by_oracle(ora, n_grid, field, cfgs)
    for method in (1, 2):
        with ps.Context(n_grid, BOX, methods=method) as ctx:
            ctx.get_FT_field(ps.PS_FIELD_DENS, field)
            B, Np, _, _ = ctx.batch(cfgs, method)
        check(method, B, Np, rB, rN)


@pytest.mark.parametrize("n_grid,count,top", [(48, 45, 23.0), (48, 3, 6.0), (60, 35, 14.0), (64, 1, 31.0)])
@pytest.mark.parametrize("kb", [0, 1, 2, 3])
def test_many_groups(gpu_lib, ora, n_grid, count, top, kb):
    """More groups than one launch takes, mixed sub-grids, lone triangles, closing
    shells that wrap; the counts by enumeration and by transforms."""
    ps = gpu_lib
    cfgs = triangles(ps, n_grid, count, top, kb, 7 * n_grid + count)
    field = synth.lognormal_density(n_grid, 2.0, 5)
    rB, rN = by_oracle(ora, n_grid, field, cfgs)
    for method in (1, 2):
        with ps.Context(n_grid, BOX, methods=method) as ctx:
            ctx.get_FT_field(ps.PS_FIELD_DENS, field)
            B, Np, _, _ = ctx.batch(cfgs, method)
            check(method, B, Np, rB, rN)
            if method == 2:
                for graph in (False, True):
                    p = ctx.plan(cfgs, method, graph=graph, fft_counts=True)
                    B2, N2, _, _ = p.execute()
                    p.close()
                    check(method, B2, N2, rB, rN)


@pytest.mark.parametrize("n_grid", [16, 48, 60])
@pytest.mark.parametrize("kb", [0, 2, 3])
def test_products_of_legs(gpu_lib, ora, n_grid, kb):
    """n = 4 to 8: powers of one leg, several distinct legs, 35 configurations, sub-grids and the whole grid."""
    ps = gpu_lib
    kf = 2 * np.pi / BOX
    top = 0.45 * n_grid
    rng = np.random.default_rng(n_grid + kb)
    sets = [[a] * 4 for a in rng.uniform(1.6, top, 3)]
    sets += [[a, a, b, b] for a, b in rng.uniform(1.6, 4.0, (3, 2))]
    sets += [list(v) for v in rng.uniform(1.6, 3.4, (20, 4))] + [list(v) for v in rng.uniform(1.6, top, (3, 4))]
    sets += [[a, a, a, b, a] for a, b in rng.uniform(1.6, 3.4, (3, 2))] + [[1.7, 2.2, 2.6] * 2] + [[1.2] * 7, [1.2] * 8]
    cfgs = []
    for s in sets:
        n = len(s)
        cfgs.append(ps.make_cfg(n, [k * kf for k in s], [0.0] * (n - 1) + [(s[-1] - 0.6) * kf],
                                [0.0] * (n - 1) + [(s[-1] + 0.8) * kf], 1.0, kb))
    field = synth.lognormal_density(n_grid, 2.0, 6)
    rB, rN = by_oracle(ora, n_grid, field, cfgs)
    for method in (1, 2):
        with ps.Context(n_grid, BOX, methods=method) as ctx:
            ctx.get_FT_field(ps.PS_FIELD_DENS, field)
            _, _, kap, _ = ctx.batch(cfgs, method, kappa=True)
            Ba, Na, _, _ = ctx.batch(cfgs, method)
            for q, g in enumerate(cfgs):
                s = slice(q, q + 1)
                check(method, Ba[s], Na[s], rB[s], rN[s], kap[s])
                B, Np, _, _ = ctx.batch([g], method)
                check(method, B, Np, rB[s], rN[s], kap[s])


# (grid, largest side): sub-grids of 60..384 points and whole grids of every length
@pytest.mark.parametrize("n_grid,top", [(96, 20.0), (128, 60.0), (192, 62.0), (256, 90.0), (300, 60.0), (320, 150.0),
                                        (384, 120.0), (512, 90.0), (600, 125.0), (600, 290.0)])
def test_transform_lengths(gpu_lib, n_grid, top):
    import torch
    ps = gpu_lib
    kf = 2 * np.pi / BOX
    torch.manual_seed(n_grid)
    field = torch.randn((n_grid,) * 3, device="cuda", dtype=torch.float32).exp_()
    top += 0.137  # no mode on an edge of a shell
    # thick shells at 1, 2/3 and 1/2 of the largest side, a square and a product of four
    sides = [[top, 0.67 * top, 0.51 * top], [0.67 * top, 0.67 * top, top], [0.8 * top] * 3, [0.12 * top] * 4, [top] * 2]
    cfgs = [ps.make_cfg(len(s), [k * kf for k in s], kbinwidth=3.0) for s in sides]
    rB, rN = by_torch(field.double(), cfgs)
    rB = np.array([float(b) for b in rB])
    torch.cuda.empty_cache()
    for method in (1, 2):
        with ps.Context(n_grid, BOX, methods=method) as ctx:
            ctx.get_FT_field(ps.PS_FIELD_DENS, field)
            _, _, kap, _ = ctx.batch(cfgs, method, kappa=True)
            Ba, Na, _, _ = ctx.batch(cfgs, method)
            for q in range(len(cfgs)):
                s = slice(q, q + 1)
                check(method, Ba[s], Na[s], rB[s], rN[s], kap[s])
                B, Np, _, _ = ctx.batch(cfgs[s], method)
                check(method, B, Np, rB[s], rN[s], kap[s])


def test_legs_beyond_the_product_memory(gpu_lib):
    """Four full-grid FP64 legs at 1024 points are above the 16 GiB of a product's spectra
    and are taken leg by leg; the FP32 legs and both counts' legs are not."""
    import torch
    ps = gpu_lib
    kf = 2 * np.pi / BOX
    torch.manual_seed(3)
    field = torch.randn((1024,) * 3, device="cuda", dtype=torch.float32).exp_()
    cfgs = [ps.make_cfg(4, [k * kf for k in (300.137, 310.21, 320.33, 200.41)], kbinwidth=0.1)]
    got = []
    for method in (1, 2):
        with ps.Context(1024, BOX, methods=method) as ctx:
            ctx.get_FT_field(ps.PS_FIELD_DENS, field)
            got.append(ctx.batch(cfgs, method, kappa=method == 2))
    (rB, rN, _, _), (B, Np, kap, _) = got
    check(2, B, Np, rB, rN, kap)


# side by side on a sub-grid (N = 64, 60), term by term on the whole grid (N = 32, 48)
@pytest.mark.parametrize("n_grid,legs", [(64, [3.3, 4.4, 5.2]), (60, [3.3, 3.3, 5.2]), (64, [4.1, 4.1, 4.1]),
                                         (32, [11.3, 12.4, 13.2]), (48, [20.3, 20.3, 20.3]), (48, [9.3, 15.1, 20.3])])
@pytest.mark.parametrize("phase", [0, 1])
def test_gradient_routes(gpu_lib, n_grid, legs, phase):
    import torch
    ps = gpu_lib
    kf = 2 * np.pi / BOX
    field = synth.lognormal_density(n_grid, 2.0, 8).astype(np.float32)
    cfg = ps.make_cfg(3, [k * kf for k in legs], kbinwidth=1.3)
    f = torch.from_numpy(field).cuda().double().requires_grad_(True)
    (B,), _ = by_torch(f, [cfg], bool(phase))
    B.backward()
    ref = f.grad.cpu().numpy()
    for method, tol in ((1, 1e-9), (2, 1e-4)):
        with ps.Context(n_grid, BOX, methods=method) as ctx:
            if phase:
                ctx.keep_modulus(True)
            ctx.get_FT_field(ps.PS_FIELD_DENS, field, use_only_phase=phase)
            g = ctx.grad(3, [k * kf for k in legs], [0.0] * 3, [0.0] * 3, 1.3, 0, method=method, double=method == 1)
        assert np.abs(g - ref).max() <= tol * np.abs(ref).max()


@pytest.mark.parametrize("bw", [0.4, 2.5])
def test_shells_without_allocation(gpu_lib, ora, bw):
    """ps_gpu_power_spectrum_noalloc with overlapping shells and gaps between them."""
    import ctypes as C

    import torch

    from test_zz_no_alloc import _dp, _noalloc
    n_grid = 32
    kf = 2 * np.pi / BOX
    ks = np.ascontiguousarray(np.linspace(1.1, 26.0, 40)[::-1] * kf)
    field = synth.lognormal_density(n_grid, 2.0, 4)
    cfgs = [gpu_lib.make_cfg(2, [k, k], kbinwidth=bw) for k in ks]
    rB, rN = by_oracle(ora, n_grid, field, cfgs)
    dev = torch.from_numpy(field).cuda()
    torch.cuda.synchronize()
    B, Np = np.zeros(len(ks)), np.zeros(len(ks))
    rc = _noalloc(gpu_lib.lib())(n_grid, float(np.float32(BOX)), C.c_void_p(dev.data_ptr()), 0, len(ks), _dp(ks), bw,
                                 _dp(B), _dp(Np), None)
    assert rc == 0
    check(2, B, Np, rB, rN)


def test_contexts_of_several_threads(gpu_lib):
    """Contexts opened, planned and closed by four threads give what one gives alone
    (plan memory passes from context to context)."""
    ps = gpu_lib
    field = synth.lognormal_density(48, 2.0, 5)
    sets = [triangles(ps, 48, 5 + 9 * t, 20.0, t % 4, t) for t in range(4)]

    def one(cfgs):
        with ps.Context(48, BOX, methods=2) as ctx:
            ctx.get_FT_field(ps.PS_FIELD_DENS, field)
            B, Np, _, _ = ctx.batch(cfgs, 2)
            p = ctx.plan(cfgs, 2)
            B2, N2, _, _ = p.execute()
            p.close()
        np.testing.assert_array_equal(N2, Np)
        np.testing.assert_array_equal(B2, B)
        return B, Np

    alone = [one(s) for s in sets]
    errors = []

    def work(t):
        try:
            for _ in range(6):
                B, Np = one(sets[t])
                np.testing.assert_array_equal(B, alone[t][0])
                np.testing.assert_array_equal(Np, alone[t][1])
        except BaseException as e:  # noqa: BLE001 - reported by the main thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(t,)) for t in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
