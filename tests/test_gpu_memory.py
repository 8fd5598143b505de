"""Device memory of a context under series of growing calls, and workspaces shared by
plans of different sizes."""
import numpy as np
import pytest

from polyspectrum_b200 import synth

pytestmark = pytest.mark.gpu

N, BOX = 256, 150.0
KF = 2 * np.pi / BOX


def used():
    import torch
    torch.cuda.synchronize()
    free, total = torch.cuda.mem_get_info()
    return total - free


def field():
    import torch
    torch.manual_seed(1)
    return torch.randn((N,) * 3, device="cuda", dtype=torch.float32).exp_()


def triangle(ps, *sides):
    return ps.make_cfg(3, [s * KF for s in sides], kbinwidth=0.5)


def spectra_bytes(method, sides):
    """Inverse transforms of the distinct legs (rows padded to 128 bytes), and the product's
    spectrum for pair groups."""
    width, size = (8, 16) if method == 1 else (16, 8)
    cols = [-(-(int(s + 0.25) + 1) // width) * width for s in sides]
    return sum(cols) * N * N * size


# two equal legs and a closing leg (FP64), three legs (FP32): sums above every sub-grid
@pytest.mark.parametrize("method,sides", [(1, (75.0,)), (2, (80.0, 81.0))])
def test_growing_calls_keep_a_bounded_workspace(gpu_lib, method, sides):
    ps = gpu_lib
    f = field()
    first = (sides * 2)[:2]
    with ps.Context(N, BOX, methods=method) as ctx:
        ctx.get_FT_field(ps.PS_FIELD_DENS, f)
        ctx.batch([triangle(ps, 20.0, 20.0, 25.0)], method)
        before = used()
        for c in np.linspace(50.0, 127.4, 60):
            _, Np, _, _ = ctx.batch([triangle(ps, *first, c)], method)
            assert Np[0] > 0
        assert used() - before <= 2 * spectra_bytes(method, (*sides, 127.4))
    # what a full-band pair of legs gives is that of a context of its own
    with ps.Context(N, BOX, methods=method) as one, ps.Context(N, BOX, methods=method) as many:
        for ctx in (one, many):
            ctx.get_FT_field(ps.PS_FIELD_DENS, f)
        for c in (60.0, 90.0, 125.0):
            B, Np, _, _ = many.batch([triangle(ps, *first, c)], method)
        B1, N1, _, _ = one.batch([triangle(ps, *first, 125.0)], method)
    np.testing.assert_array_equal(Np, N1)
    np.testing.assert_array_equal(B, B1)


def test_one_full_band_leg_fits_the_work_spectrum(gpu_lib):
    ps = gpu_lib
    with ps.Context(N, BOX, methods=1) as ctx:
        ctx.get_FT_field(ps.PS_FIELD_DENS, field())
        ctx.batch([triangle(ps, 20.0, 20.0, 20.0)], 1)
        before = used()
        ctx.batch([triangle(ps, 128.1, 128.1, 128.1)], 1)  # band 128
        assert used() - before <= 32 << 20


def test_growing_shell_lists_keep_bounded_sums(gpu_lib):
    ps = gpu_lib
    n = 128
    with ps.Context(n, BOX, methods=2) as ctx:
        ctx.get_FT_field(ps.PS_FIELD_DENS, synth.lognormal_density(n, 2.0, 3))
        ks = np.linspace(1.0, 63.0, 1600) * KF
        cfgs = [ps.make_cfg(2, [k, k], kbinwidth=1.0) for k in ks]
        ctx.batch(cfgs[:4], 2)
        before = used()
        for m in range(16, 1601, 16):
            ctx.batch(cfgs[:m], 2)
        assert used() - before <= 16 << 20


@pytest.mark.parametrize("graph", [False, True])
def test_plans_keep_their_workspace(gpu_lib, graph):
    """A plan runs on after larger calls have replaced the workspace it was made with;
    the memory goes with the last plan that holds it."""
    ps = gpu_lib
    with ps.Context(N, BOX, methods=2) as ctx:
        ctx.get_FT_field(ps.PS_FIELD_DENS, field())
        small = [triangle(ps, 80.0, 81.0, 50.0), ps.make_cfg(4, [k * KF for k in (60.0, 61.0, 62.0, 63.0)])]
        large = [triangle(ps, 80.0, 81.0, 127.4), ps.make_cfg(4, [k * KF for k in (100.0, 101.0, 102.0, 110.0)])]
        p = ctx.plan(small, graph=graph)
        want = p.execute()
        q = ctx.plan(large, graph=graph)
        wantq = q.execute()
        held = used()
        for _ in range(2):
            for plan, w in ((p, want), (q, wantq)):
                B, Np, _, _ = plan.execute()
                np.testing.assert_array_equal(Np, w[1])
                np.testing.assert_array_equal(B, w[0])
        p.close()
        assert used() < held - (100 << 20)
        B, Np, _, _ = q.execute()
        np.testing.assert_array_equal(Np, wantq[1])
        np.testing.assert_array_equal(B, wantq[0])
        q.close()


def test_calls_after_running_out_of_memory(gpu_lib):
    """A refused allocation is that call's error and no later one's."""
    import torch
    ps = gpu_lib
    with ps.Context(N, BOX) as ctx:
        ctx.get_FT_field(ps.PS_FIELD_DENS, field())
        small, large = [triangle(ps, 20.0, 21.0, 25.0)], [triangle(ps, 100.0, 101.0, 127.4)]
        want = ctx.batch(small, 2)
        wantp = ctx.batch(small, 1)
        torch.cuda.empty_cache()
        hog = torch.empty(torch.cuda.mem_get_info()[0] - (48 << 20), dtype=torch.uint8, device="cuda")
        for refused in (lambda: ctx.batch(large, 2), lambda: ctx.batch(large, 1), lambda: ps.Context(N, BOX),
                        lambda: ctx.grad(3, [20 * KF] * 3, [0.0] * 3, [0.0] * 3, 0.5, 0)):
            with pytest.raises(ps.PsError) as err:
                refused()
            assert err.value.status == -2, err.value
            for method, w in ((2, want), (1, wantp)):
                B, Np, _, _ = ctx.batch(small, method)
                np.testing.assert_array_equal(Np, w[1])
                np.testing.assert_array_equal(B, w[0])
        del hog
        torch.cuda.empty_cache()
        _, Np, _, _ = ctx.batch(large, 2)
        assert Np[0] > 0
