"""Work on a context between ps_gpu_plan_prepare of counts by FP64 transforms, which
stay on the side stream, and their plan's execution: everybody's results are those of
the calls made one after the other."""
import numpy as np
import pytest

from polyspectrum_b200 import synth

pytestmark = pytest.mark.gpu

N, BOX = 128, 150.0
KF = 2 * np.pi / BOX


def triangles(ps, kb, count, top, seed):
    rng = np.random.default_rng(seed)
    cfgs = []
    for a in rng.uniform(0.5 * top, top, count):
        cfgs.append(ps.make_cfg(3, [a * KF, a * KF, 0.8 * a * KF], [0.0, 0.0, (0.8 * a - 0.4) * KF],
                                [0.0, 0.0, (0.8 * a + 0.7) * KF], 1.0, kb))
    return cfgs


def quads(ps):
    rng = np.random.default_rng(5)
    return [ps.make_cfg(4, [k * KF for k in s]) for s in rng.uniform(2.0, 25.0, (6, 4))]


def same(got, want):
    np.testing.assert_array_equal(got[1], want[1])
    np.testing.assert_array_equal(got[0], want[0])


@pytest.mark.parametrize("graph", [False, True])
def test_work_between_prepare_and_execution(gpu_lib, graph):
    import torch
    ps = gpu_lib
    field = torch.from_numpy(synth.lognormal_density(N, 2.0, 3)).cuda()
    long = triangles(ps, ps.PS_BIN_WATKINSON, 24, 42.0, 1)  # several ms of counts on the side stream
    mixed = triangles(ps, ps.PS_BIN_WATKINSON, 2, 12.0, 2) + quads(ps)
    leg = [9.0 * KF, 11.0 * KF, 13.0 * KF]
    with ps.Context(N, BOX) as ctx:
        ctx.get_FT_field(ps.PS_FIELD_DENS, field)
        p, q = ctx.plan(long, graph=graph), ctx.plan(mixed, graph=graph)
        products = ctx.plan(quads(ps), graph=graph)
        g = torch.empty(N, N, N, dtype=torch.float64, device="cuda")

        def gradient():
            ctx.grad(3, leg, [0.0] * 3, [0.0] * 3, 1.0, 0, out=g)
            return g.cpu().numpy(), np.zeros(1)

        def prepared():
            q.prepare()
            p.prepare()  # (already prepared by the caller: nothing more)
            return q.execute()

        work = {"batch": lambda: ctx.batch(quads(ps)), "plan": products.execute, "fft plan": q.execute,
                "plain": lambda: ctx.batch(quads(ps), ps.PS_FP64_PLAIN), "gradient": gradient, "prepared": prepared}
        alone = {name: f() for name, f in work.items()}
        want = p.execute()
        assert (want[1] > 0).all()
        for name, f in work.items():
            for _ in range(3):
                p.prepare()
                same(f(), alone[name])
                same(p.execute(), want)
        # a plan prepared first, counts of another behind it
        for _ in range(3):
            q.prepare()
            p.prepare()
            same(q.execute(), alone["fft plan"])
            same(p.execute(), want)
        for plan in (p, q, products):
            plan.close()


def test_tuning_between_prepare_and_execution(gpu_lib):
    ps = gpu_lib
    field = synth.lognormal_density(N, 2.0, 3)
    with ps.Context(N, BOX, methods=ps.PS_FP32_BATCHED) as ctx:
        ctx.get_FT_field(ps.PS_FIELD_DENS, field)
        p = ctx.plan(triangles(ps, ps.PS_BIN_WATKINSON, 24, 42.0, 1))
        want = p.execute()[1]
        p.prepare()
        q = ctx.plan(triangles(ps, ps.PS_BIN_WATKINSON, 4, 36.0, 7), autotune=True)  # times FP64 counts
        np.testing.assert_array_equal(p.execute()[1], want)
        tuned = q.execute()[1]
        q.close()
        p.close()
    with ps.Context(N, BOX, methods=ps.PS_FP32_BATCHED) as ctx:
        ctx.get_FT_field(ps.PS_FIELD_DENS, field)
        np.testing.assert_array_equal(ctx.batch(triangles(ps, ps.PS_BIN_WATKINSON, 4, 36.0, 7))[1], tuned)


def test_plan_destroyed_while_a_callers_stream_still_runs_it(gpu_lib):
    """A launch and its result copy queued on a caller's stream, the context given back to
    its own stream, the plan destroyed and others made in its memory: the copy still
    brings the first plan's results."""
    import torch
    ps = gpu_lib
    field = torch.from_numpy(synth.lognormal_density(N, 2.0, 3)).cuda()
    first, other = triangles(ps, 0, 6, 30.0, 1), triangles(ps, 0, 9, 20.0, 2)
    s = torch.cuda.Stream()
    with ps.Context(N, BOX, methods=ps.PS_FP32_BATCHED) as ctx:
        ctx.get_FT_field(ps.PS_FIELD_DENS, field)
        for graph in (False, True):
            p = ctx.plan(first, graph=graph)
            B, Np, _, _ = p.execute()
            out = torch.zeros(8 * len(first), dtype=torch.float64, device="cuda")
            torch.cuda.synchronize()
            with torch.cuda.stream(s):
                torch.cuda._sleep(100_000_000)  # some 50 ms ahead of the launch
            ctx.set_stream(s.cuda_stream)
            p.launch()
            p.results_to_device(out.data_ptr())
            ctx.set_stream(None)
            p.close()
            for _ in range(4):
                q = ctx.plan(other, graph=graph)
                q.execute()
                q.close()
            torch.cuda.synchronize()
            got = out.cpu().numpy()[:2 * len(first)].reshape(-1, 2)
            np.testing.assert_array_equal(got[:, 0], B)
            np.testing.assert_array_equal(got[:, 1], Np)


def test_launch_inside_a_callers_graph(gpu_lib):
    """An eager plan launched on a caller's stream that captures: the caller's graph
    replays it on the field loaded last."""
    import torch
    ps = gpu_lib
    fields = [torch.from_numpy(synth.lognormal_density(N, 2.0, seed)).cuda() for seed in (3, 4)]
    cfgs = triangles(ps, 0, 6, 30.0, 1) + triangles(ps, ps.PS_BIN_WATKINSON, 2, 12.0, 2) + quads(ps)
    with ps.Context(N, BOX, methods=ps.PS_FP32_BATCHED) as ctx:
        p = ctx.plan(cfgs, graph=False)
        want = []
        for f in fields:
            ctx.get_FT_field(ps.PS_FIELD_DENS, f)
            want.append(p.execute()[:2])
        p.prepare()  # counts by transforms have been on the side stream of this context
        p.execute()
        s = torch.cuda.Stream()
        ctx.set_stream(s.cuda_stream)
        p.launch()  # one launch outside: the capture below finds everything made
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            p.launch()
        ctx.set_stream(None)
        for f, w in zip(fields, want):
            ctx.get_FT_field(ps.PS_FIELD_DENS, f)
            g.replay()
            torch.cuda.synchronize()
            same(p.results()[:2], w)
        p.close()
