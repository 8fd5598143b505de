"""Timed cases of the polyspectrum estimator, each through the calls a user's program makes.

A case names a call pattern and a workload:

  call    noalloc  ps_gpu_power_spectrum_noalloc on a device field (host programs that may not allocate)
          batch    load the field, then evaluate the configuration list once (Context.batch), as a script with
                   one field and one list does; planning is part of the call
          plan     a plan made once, then per field of a series: load, execute
          series   the plan with its field-independent parts queued ahead of the load (Plan.prepare), no
                   read-back before the results are fetched
          grad     autograd: B of one configuration and its gradient with respect to the field
  shape   power (n = 2, all shells), equilateral (n = 3), theta (n = 3, sweeps over the pairs of `legs`),
          triangles (equilateral + one theta sweep), polygons (n = legs per configuration, DEFAULT binning)
  legs    k values in h/Mpc, "k1,k2;k1,k2;..." (one configuration per ';' for polygons)
  source  device, pinned or pageable: where the input grid lies when the call is made
  method  1 PS_FP64_PLAIN, 2 PS_FP32_BATCHED

Sizes, boxes, spectra and binnings are those of the named configurations (128^3 L = 200, 256^3 L = 300,
512^3 L = 400, 600^3, 1024^3 L = 1000), of the tests and of the benchmark.

Bispectra and power spectra of the FP32 method are returned in single precision, which is what its transforms
and its error estimate (condition number times 2^-24) give; those of the FP64 method in double precision.  Polygon
counts of the batched method are integers.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

import polyspectrum_b200 as ps
from polyspectrum_b200 import autograd as ps_autograd

BW = 1.0  # kbinwidth of every configuration (the reference's default)
DCOS = 0.1  # cosThetaBinwidth of GIVEN / WATKINSON sweeps


def listed():
    return [
        # the smallest call: a monitoring P(k) of a 64^3 field inside a simulation step
        dict(name="power_64_noalloc", call="noalloc", grid=64, box=150.0, field="dens", phase=0, source="device",
             shape="power", n=2, values=32, legs="", binning=0, method=2),
        # a small mixed-radix grid evaluated once, planning included: a test-size run of the driver loop
        dict(name="theta_48_batch", call="batch", grid=48, box=150.0, field="xhi_dens", phase=0, source="device",
             shape="theta", n=3, values=8, legs="0.15,0.22", binning=1, method=2),
        # trispectrum configurations (n = 4), evaluated leg by leg, from a pageable host array
        dict(name="polygons_96", call="batch", grid=96, box=150.0, field="dens", phase=0, source="pageable",
             shape="polygons", n=4, values=6, legs="0.3,0.3,0.4,0.5;0.2,0.3,0.3,0.4;0.5,0.5,0.5,0.5;0.25,0.45,0.5,0.6;"
             "0.6,0.3,0.6,0.3;0.35,0.4,0.45,0.5", binning=0, method=2),
        # the 128^3 configuration's equilateral sweep, repeated over a series of fields
        dict(name="equilateral_128", call="plan", grid=128, box=200.0, field="dens", phase=0, source="device",
             shape="equilateral", n=3, values=64, legs="", binning=0, method=2),
        # the same configuration as the reference computes it: FP64, one configuration at a time
        dict(name="equilateral_128_fp64", call="batch", grid=128, box=200.0, field="dens", phase=0, source="device",
             shape="equilateral", n=3, values=64, legs="", binning=0, method=1),
        # WATKINSON shells are no radius intervals: counts come from FP64 transforms
        dict(name="watkinson_192", call="plan", grid=192, box=250.0, field="xhii", phase=0, source="device",
             shape="theta", n=3, values=12, legs="0.4,0.7;0.6,0.6", binning=3, method=2),
        # the 256^3 ionisation map, GIVEN binning, 20 angles, one field read into pinned host memory
        dict(name="given_256", call="batch", grid=256, box=300.0, field="xhii", phase=0, source="pinned",
             shape="theta", n=3, values=20, legs="0.5,1.0", binning=2, method=2),
        # the adjoint configuration (equilateral k = 0.8 at 256^3): FP64 forward and backward
        dict(name="grad_256_fp64", call="grad", grid=256, box=200.0, field="dens", phase=0, source="device",
             shape="polygons", n=3, values=1, legs="0.8,0.8,0.8", binning=0, method=1),
        # a scalene triangle through the phase normalisation: FP32 forward and backward
        dict(name="grad_256_phase", call="grad", grid=256, box=200.0, field="dens", phase=1, source="device",
             shape="polygons", n=3, values=1, legs="0.5,0.7,0.9", binning=0, method=2),
        # the headline workload: 512^3 phase-only field, 64 DERIVED configurations on a series of fields
        dict(name="sweep_512", call="series", grid=512, box=400.0, field="xhi_dens", phase=1, source="device",
             shape="theta", n=3, values=16, legs="0.2,0.5;0.5,0.8;0.8,1.2;1.0,1.5", binning=1, method=2),
        # equilateral triangles up to Nyquist and an isosceles sweep on the 600^3 grid of the accuracy study
        dict(name="triangles_600", call="plan", grid=600, box=600.0, field="dens", phase=0, source="device",
             shape="triangles", n=3, values=32, legs="0.3,0.3", binning=0, method=2),
        # the large grid: all 512 shells of the power spectrum at 1024^3
        dict(name="power_1024", call="plan", grid=1024, box=1000.0, field="dens", phase=0, source="device",
             shape="power", n=2, values=512, legs="", binning=0, method=2),
    ]


def _sizes(rng, lo, hi):
    """A supported grid size of [lo, hi], spread over its logarithm."""
    want = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    sizes = [q for q in (16, 32, 48, 60, 64, 96, 128, 192, 256, 300, 320, 384, 512, 600, 1024) if lo <= q <= hi]
    return min(sizes, key=lambda q: abs(math.log(q / want)))


def draw(rng):
    """One more case: any call on any supported grid of the range its cost allows."""
    call = rng.choice(["noalloc", "batch", "batch", "plan", "plan", "series", "grad"])
    method, shape, n, binning = 2, "theta", 3, 0
    if call == "noalloc":
        grid, shape, n = rng.choice([16, 32, 64]), "power", 2
    elif call == "grad":
        grid, shape, method = _sizes(rng, 32, 384), "polygons", rng.choice([1, 2])
    else:
        method = rng.choice([1, 2, 2, 2, 2]) if call == "batch" else 2
        shape = rng.choice(["power", "equilateral", "theta", "theta", "triangles", "polygons"])
        grid = _sizes(rng, 32, 192 if method == 1 or shape == "polygons" else 600)
        if shape == "theta":
            binning = rng.choice([0, 1, 2, 3])
            if binning == 3:
                grid = min(grid, 256)
        n = 2 if shape == "power" else rng.choice([3, 4, 5]) if shape == "polygons" else 3
    field = rng.choice(["dens", "xhii", "xhi_dens"]) if call in ("batch", "plan", "series") else "dens"
    box = round(rng.uniform(0.6, 1.6) * grid, 2)
    kf = 2 * math.pi / box
    top = 0.22 * grid  # every triangle of the sweep keeps its closing leg near or below Nyquist
    k = lambda: round(kf * rng.uniform(2.5, top), 5)  # noqa: E731
    values, legs = rng.randint(2, 24), ""
    if shape == "power":
        values = grid // 2 if call != "noalloc" else rng.randint(4, grid // 2)
    elif shape == "theta":
        legs = ";".join("%r,%r" % (k(), k()) for _ in range(rng.randint(1, 4)))
    elif shape == "triangles":
        k1 = k()
        legs = "%r,%r" % (k1, k1)
    elif shape == "polygons":
        values = 1 if call == "grad" else rng.randint(1, 8)
        legs = ";".join(_polygon(rng, n, kf, top) for _ in range(values))
    source = rng.choice(["device", "device", "pinned", "pageable"]) if call == "batch" else "device"
    phase = 0 if n == 2 else rng.choice([0, 0, 1])  # a phase-only power spectrum is the same for every field
    return dict(call=call, grid=grid, box=box, field=field, phase=phase, source=source, shape=shape, n=n,
                values=values, legs=legs, binning=binning, method=method)


def _polygon(rng, n, kf, top):
    """Legs of one closed polygon: all within a factor of two, so the longest is below the others' sum."""
    lo = rng.uniform(2.5, top / 2 if top > 5 else 2.6)
    return ",".join("%r" % round(kf * lo * rng.uniform(1.0, 1.8), 5) for _ in range(n))


# ---------------------------------------------------------------- inputs
def _gaussian(n, alpha, seed):
    """Unit-variance Gaussian field with P(k) ~ k^-alpha up to Nyquist (polyspectrum_b200/synth.py's recipe)."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    w = torch.fft.rfftn(torch.randn((n, n, n), generator=g, device="cuda"))
    f = torch.fft.fftfreq(n, device="cuda") * n
    z = torch.fft.rfftfreq(n, device="cuda") * n
    for i in range(n):  # plane by plane: no further array of the grid's size
        k2 = f[i] ** 2 + f[:, None] ** 2 + z[None, :] ** 2
        w[i] *= torch.where((k2 > 0) & (k2 <= (n / 2) ** 2), k2.clamp_min(1.0) ** (-alpha / 4.0), torch.zeros_like(k2))
    r = torch.fft.irfftn(w, s=(n, n, n))
    r /= r.std()
    return r


def _inputs(case, seed):
    """(density, x_HII) grids of the case's field, None where it uses none."""
    n, dens, xhii = case["grid"], None, None
    if case["field"] in ("dens", "xhi_dens"):
        dens = torch.exp(_gaussian(n, 1.5 if n >= 600 else 2.0, 2 * seed) - 0.5)
        if case["field"] == "dens":
            dens -= 1.0  # lognormal contrast; the XHI_DENS product takes the density 1 + delta
    if case["field"] in ("xhii", "xhi_dens"):
        # binary ionisation map: the connected regions where a smooth field is high
        xhii = (_gaussian(n, 3.0, 2 * seed + 1) > 0.6).float()
    torch.cuda.empty_cache()
    return dens, xhii


def _pairs(case):
    return [tuple(float(v) for v in p.split(",")) for p in case["legs"].split(";")] if case["legs"] else []


def _configs(case):
    N, L = case["grid"], case["box"]
    if case["shape"] == "polygons":
        return [ps.make_cfg(case["n"], list(p), kbinwidth=BW, kbinningCase=case["binning"]) for p in _pairs(case)]
    out = []
    if case["shape"] == "power":
        out += list(ps.read_params_to_kvectors(N, L, 2, num_values=2, kbinwidth=BW)[0])
    if case["shape"] in ("equilateral", "triangles"):
        out += list(ps.read_params_to_kvectors(N, L, 3, equilateral=1, num_values=case["values"], kbinwidth=BW)[0])
    for k1, k2 in _pairs(case):
        out += list(ps.read_params_to_kvectors(N, L, 3, k1=k1, k2=k2, num_values=case["values"], kbinwidth=BW,
                                               kbinningCase=case["binning"], dcosTheta=DCOS)[0])
    return out


FIELDS = {"dens": ps.PS_FIELD_DENS, "xhii": ps.PS_FIELD_XHII, "xhi_dens": ps.PS_FIELD_XHI_DENS}


def prepare(case, seed):
    dens, xhii = _inputs(case, seed)
    s = dict(case=dict(case), dens=dens, xhii=xhii)
    if case["call"] == "noalloc":
        f = ps.lib().ps_gpu_power_spectrum_noalloc
        dp = C.POINTER(C.c_double)
        f.argtypes = [C.c_int, C.c_double, C.c_void_p, C.c_int, C.c_int, dp, C.c_double, dp, dp, C.c_void_p]
        f.restype = C.c_int
        s["fn"], s["L"], s["k"] = f, float(np.float32(case["box"])), _power_k(case)
        return s
    if case["source"] != "device":
        host = lambda t: None if t is None else t.cpu().pin_memory() if case["source"] == "pinned" else t.cpu().numpy()  # noqa: E731
        s["dens"], s["xhii"] = host(dens), host(xhii)
        del dens, xhii
        torch.cuda.empty_cache()
    cfgs = _configs(case)
    s["cfgs"] = (ps.ps_cfg * len(cfgs))(*cfgs)
    s["ctx"] = ctx = ps.Context(case["grid"], case["box"], methods=case["method"])
    if case["call"] in ("plan", "series"):
        s["plan"] = ctx.plan(s["cfgs"], graph=True, autotune=True)
        if case["call"] == "series":
            ctx.set_spectrum_band(s["plan"].band)
    if case["call"] == "grad":
        s["dens"] = (dens.double() if case["method"] == 1 else dens).requires_grad_()
    return s


def _power_k(case):
    return 2 * math.pi / float(np.float32(case["box"])) * np.arange(1, case["values"] + 1, dtype=np.float64)


def _ranges(cfgs):
    """kmin, kmax of every configuration (as DERIVED binning writes them back)."""
    return np.frombuffer(cfgs, dtype=np.float64).reshape(len(cfgs), C.sizeof(ps.ps_cfg) // 8)[:, -2 * ps.PS_MAX_LEGS:].copy()


# ---------------------------------------------------------------- one pass
def run(s):
    case = s["case"]
    which, phase = FIELDS[case["field"]], case["phase"]
    if case["call"] == "noalloc":
        k = s["k"]
        P, Np = np.zeros(len(k)), np.zeros(len(k))
        dp = lambda a: a.ctypes.data_as(C.POINTER(C.c_double))  # noqa: E731
        rc = s["fn"](case["grid"], s["L"], s["dens"].data_ptr(), phase, len(k), dp(k), BW, dp(P), dp(Np), None)
        if rc != 0:
            raise RuntimeError("status %d" % rc)
        return {"B": P.astype(np.float32), "npoly": Np.astype(np.int64)}
    ctx = s["ctx"]
    if case["call"] == "grad":
        f = s["dens"]
        B = ps_autograd.polyspectrum(f, ctx, s["cfgs"][0], case["method"], phase)
        (g,) = torch.autograd.grad(B, f)
        return {"B": B if case["method"] == 1 else B.float(), "grad": g}
    if case["call"] == "batch":
        ctx.get_FT_field(which, s["dens"], s["xhii"], use_only_phase=phase)
        B, Np, _, cfgs = ctx.batch(s["cfgs"], case["method"])
    elif case["call"] == "plan":
        ctx.get_FT_field(which, s["dens"], s["xhii"], use_only_phase=phase)
        B, Np, _, cfgs = s["plan"].execute()
    else:
        s["plan"].prepare()
        ctx.set_field_async(which, s["dens"], s["xhii"], use_only_phase=phase)
        s["plan"].launch()
        B, Np, _, cfgs = s["plan"].results()
    if case["method"] == 2:
        return {"B": B.astype(np.float32), "npoly": Np.astype(np.int64), "ranges": _ranges(cfgs)}
    return {"B": B, "npoly": Np, "ranges": _ranges(cfgs)}


# ---------------------------------------------------------------- work
def _legs_of(case):
    """(k, kmin, kmax) lists of every configuration: kvectors.c:75-137 with the GIVEN ranges of run.c:56-84."""
    N, L, pi = case["grid"], case["box"], math.pi
    if case["shape"] == "polygons":
        return [(list(p), [0.0] * len(p), [0.0] * len(p)) for p in _pairs(case)]
    if case["call"] == "noalloc":
        return [([k, k], [0.0] * 2, [0.0] * 2) for k in _power_k(case)]
    out = []
    if case["shape"] == "power":
        out += [([2.0 * pi / L * (i + 1.0)] * 2, [0.0] * 2, [0.0] * 2) for i in range(N // 2)]
    if case["shape"] in ("equilateral", "triangles"):
        ks = [2.0 * pi / L * math.pow(N // 2, (i + 1.0) / case["values"]) for i in range(case["values"])]
        out += [([k] * 3, [0.0] * 3, [0.0] * 3) for k in ks]
    for k1, k2 in _pairs(case):
        for i in range(case["values"]):
            th = pi * i / case["values"]
            side = lambda c: math.sqrt(k1 * k1 + k2 * k2 - 2.0 * k1 * k2 * c)  # noqa: E731
            lo, hi = [0.0] * 3, [0.0] * 3
            if case["binning"] >= 2:
                lo[2] = side(min(1.0, math.cos(th) + 0.5 * DCOS))
                hi[2] = side(max(-1.0, math.cos(th) - 0.5 * DCOS))
            out.append(([k1, k2, side(math.cos(th))], lo, hi))
    return out


def work(case):
    """Bytes: every input grid read once, the gradient written once, a few numbers per configuration.  Flops: the
    forward transform of the field, and per distinct set of legs one transform of each leg and one of the product on
    the smallest grid that holds the polygon without wrap-around (2.5 M^3 log2 M^3 each)."""
    N = case["grid"]
    wide = 8.0 if case["call"] == "grad" and case["method"] == 1 else 4.0
    legs = _legs_of(case)
    nbytes = wide * N ** 3 * (2 if case["field"] == "xhi_dens" else 1) + 200.0 * len(legs)
    fft = lambda m: 2.5 * m ** 3 * 3 * math.log2(max(m, 2))  # noqa: E731
    flops = fft(N)
    if case["n"] > 2:
        kf, seen = 2 * math.pi / case["box"], set()
        for k, _, _ in legs:
            first = tuple(sorted(k[:2])) if case["n"] == 3 else tuple(sorted(k))
            if first not in seen:
                seen.add(first)
                m = min(N, int(2 * sum(sorted(first)) / kf) + 4 if case["n"] == 3 else int(sum(first) / kf) + 4)
                flops += (len(set(first)) + 1) * fft(m)
    else:
        flops += 4.0 * N ** 3 / 2
    if case["call"] == "grad":
        nbytes += wide * N ** 3
        flops += fft(N)
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------- the same numbers in 64 bits
class _Exact:
    """The estimator by its definition (polyspectrum.c:51-252) with torch in FP64."""

    def __init__(self, case, seed):
        self.case, self.N = case, case["grid"]
        self.L = float(np.float32(case["box"]))
        dens, xhii = _inputs(case, seed)
        f = {"dens": lambda: dens.double(), "xhii": lambda: xhii.double(),
             "xhi_dens": lambda: dens.double() * (1.0 - xhii.double())}[case["field"]]()
        del dens, xhii
        self.field = f.requires_grad_() if case["call"] == "grad" else f
        self.dk = torch.fft.rfftn(self.field)
        if case["call"] != "grad":
            self.field = None
        if case["phase"]:
            self.dk = self.dk / self.dk.abs()
        m = np.arange(self.N)
        m = torch.from_numpy(np.where(m < self.N // 2, m, m - self.N)).cuda()
        self.m, self.h = m, m[: self.N // 2 + 1].abs()

    def r2(self, i):
        """|m|^2 of the planes i of the half spectrum."""
        return (self.m[i, None, None] ** 2 + self.m[None, :, None] ** 2 + self.h[None, None, :] ** 2).int()

    def corners(self):
        """Smallest and largest squared corner radius of every mode's cell (get_corners, filter.c:257-289)."""
        e = 0.5 * BW
        one = lambda x: ((x.double() - e) * (x.double() - e), (x.double() + e) * (x.double() + e))  # noqa: E731
        ax = [one(self.m), one(self.m), one(self.h)]
        out = []
        for pick in (torch.minimum, torch.maximum):
            x, y, z = (pick(*a) for a in ax)
            out.append((x[:, None, None] + y[None, :, None]) + z[None, None, :])
        return out

    def scale(self, k):
        return k / (2.0 * math.pi) * self.L

    def table(self, lower, upper):
        """Whether each |m|^2 has lower(|m|) and upper(|m|)."""
        s = np.sqrt(np.arange(3 * (self.N // 2) ** 2 + 1, dtype=np.float64))
        return torch.from_numpy(lower(s) & upper(s)).cuda()

    def mask(self, kind, k, lo=0.0, hi=0.0):
        half, kk, a, b = 0.5 * BW, self.scale(k), self.scale(lo), self.scale(hi)
        if kind < 2:
            t = (self.table(lambda s: kk - s <= half, lambda s: kk - s >= -half) if kind == 0
                 else self.table(lambda s: a - s <= half, lambda s: s - b <= half))
            return torch.cat([t[self.r2(slice(i, i + 32)).long()] for i in range(0, self.N, 32)])
        p, q = (c.sqrt() for c in self.corners())
        if kind == 2:
            return (p <= kk) & (kk <= q)
        return ((q >= b) & (p <= b)) | ((q <= b) & (p >= a)) | ((q >= a) & (p <= a))

    def shells(self, k, lo, hi):
        """Masks of a configuration's legs, with the DERIVED ranges written into lo and hi."""
        n, b = len(k), self.case["binning"]
        if b == 0:
            return [(0, v, 0.0, 0.0) for v in k]
        if b == 1:
            for j in range(2):
                if (k[j],) not in self.kept:
                    inside = self.mask(0, k[j])
                    p, q = self.corners()
                    self.kept[(k[j],)] = (float(p[inside].min()), float(q[inside].max()))
                p, q = self.kept[(k[j],)]
                lo[j], hi[j] = (math.sqrt(v) * 2.0 * math.pi / self.L for v in (p, q))
            c = (k[0] * k[0] + k[1] * k[1] - k[2] * k[2]) / (2.0 * k[0] * k[1])
            t = [x * x + y * y - 2.0 * x * y * c for x, y in
                 [(lo[0], lo[1]), (lo[0], hi[1]), (hi[0], lo[1]), (hi[0], hi[1]), (k[0], hi[1]), (hi[0], k[1]),
                  (k[0], lo[1]), (lo[0], k[1])]]
            lo[2], hi[2] = math.sqrt(min(t)), math.sqrt(max(t))
        first = 2 if b == 3 else 0
        return [(first, v, 0.0, 0.0) for v in k[: n - 1]] + [(first + 1, k[-1], lo[-1], hi[-1])]

    def real(self, key, spectrum):
        """Unnormalised inverse transforms of a shell of the field (or of the shell itself)."""
        F = self.mask(*key)
        return torch.fft.irfftn(F.to(torch.complex128) if spectrum is None else F * spectrum, s=(self.N,) * 3, norm="forward")

    def all(self):
        N, n, legs = self.N, self.case["n"], _legs_of(self.case)
        V = self.L ** 3
        coef = V ** (n - 1) * float(N) ** (-3 * n)
        B, cnt, ranges, self.kept, fields = [], [], np.zeros((len(legs), 2 * ps.PS_MAX_LEGS)), {}, {}
        if n == 2:
            size = 3 * (N // 2) ** 2 + 1
            S, W = torch.zeros(size, dtype=torch.float64, device="cuda"), torch.zeros(size, dtype=torch.float64, device="cuda")
            w = torch.full((N // 2 + 1,), 2.0, dtype=torch.float64, device="cuda")
            w[0] = w[-1] = 1.0
            for i in range(0, N, 16):
                r = self.r2(slice(i, i + 16)).reshape(-1)
                d = self.dk[i: i + 16]
                S += torch.bincount(r, ((d.real ** 2 + d.imag ** 2) * w).reshape(-1), minlength=size)
                W += torch.bincount(r, w.expand(d.shape).reshape(-1), minlength=size)
        for q, (k, lo, hi) in enumerate(legs):
            if n == 2:
                kk = self.scale(k[0])
                t = self.table(lambda s: kk - s <= 0.5 * BW, lambda s: kk - s >= -0.5 * BW)
                sd, si = float(N) ** 3 * float(S[t].sum()), float(N) ** 3 * float(W[t].sum())
            else:
                keys = self.shells(k, lo, hi)
                for key in keys[: n - 1]:
                    if key not in fields:
                        if len(fields) >= 3:
                            fields.pop(next(iter(fields)))
                        fields[key] = (self.real(key, self.dk), self.real(key, None))
                last = fields[keys[-1]] if keys[-1] in fields else (self.real(keys[-1], self.dk), self.real(keys[-1], None))
                D, I = last
                for key in keys[: n - 1]:
                    D, I = D * fields[key][0], I * fields[key][1]
                sd, si = D.sum(), float(I.sum())
                if self.field is None:
                    sd = float(sd)
            cnt.append(round(si / float(N) ** 3))
            B.append(coef * sd / (cnt[-1] * float(N) ** 3))
            ranges[q, : len(lo)], ranges[q, ps.PS_MAX_LEGS: ps.PS_MAX_LEGS + len(hi)] = lo, hi
        return B, cnt, ranges


def exact(case, seed):
    e = _Exact(case, seed)
    B, cnt, ranges = e.all()
    if case["call"] == "grad":
        (g,) = torch.autograd.grad(B[0], e.field)
        return {"B": B[0].detach(), "grad": g}
    out = {"B": np.array(B), "npoly": np.array(cnt, dtype=np.float64 if case["method"] == 1 else np.int64)}
    if case["call"] != "noalloc":
        out["ranges"] = ranges
    return out
