"""The work that is measured: gridding, degridding and imaging calls over their real range.

``listed()`` holds the named cases, ``draw()`` gives more of the same ranges,
``prepare()`` makes a case's inputs from a seed, ``run()`` is one pass through the
public entry points, ``work()`` says what a pass cannot do without and ``exact()``
what it returns in 64 bits, in plain torch.

The kinds:

  conv       conv_imaging + conv_predict with a caller's kernel (separable or 4-D)
  driver     do_imaging + do_predict, host arrays in and out, as the reference is called
  wproj      w_cache_imaging + w_cache_predict: w-projection both ways
  diff       predicted visibilities of an image and the gradient of their misfit
  aw         AW-projection of a batch: plan, grid, degrid (the headline workload)
  aw_cycle   a major cycle's plan and fused degrid + residual grid pass
  aw_table   generation of a table of AW kernels
  wstack     w_stack_imaging: every plane gridded, transformed and combined
  wtowers    w_towers_imaging + w_towers_predict
  recombine  facets to subgrids and back
"""

import math

import numpy
import torch

from crocodile_gb300 import autograd, awproj, engine, recombine, synthesis

C64, C128, F64 = torch.complex64, torch.complex128, torch.float64


def listed():
    return [
        # the smallest imaging calls: a snapshot, or one facet of many; latency counts
        dict(name="conv_snapshot", kind="conv", N=256, n=1000, S=8, Q=8, sep=True, precision="fp32"),
        # one channel of a full 4-D kernel at an odd size
        dict(name="conv_odd", kind="conv", N=1531, n=123457, S=9, Q=4, sep=False, precision="fp32"),
        # the reference's own call on host arrays, at its usual size
        dict(name="driver_1024", kind="driver", N=1024, n=200000, S=8, Q=8),
        # the plain complex128 form, used to check results
        dict(name="wproj_fp64", kind="wproj", N=1024, n=50000, S=9, Q=4, wrange=300.0, wstep=20.0,
             npixff=32, precision="fp64"),
        # w-projection of a wide field
        dict(name="wproj_4096", kind="wproj", N=4096, n=2000000, S=15, Q=8, wrange=500.0,
             wstep=10.0, npixff=64, precision="fp32"),
        # one step of a fit to visibilities: forward and backward
        dict(name="diff_2048", kind="diff", N=2048, n=1000000, S=8, Q=8),
        # a major cycle of a mid-sized array
        dict(name="aw_cycle_4096", kind="aw_cycle", N=4096, nant=32, ntime=63, nchan=64, wbins=32),
        # the whole AW data set: 64 antennas, 16.1M visibilities
        dict(name="aw_8192", kind="aw", N=8192, nant=64, ntime=125, nchan=64, wbins=64),
        # AW kernels of a new data set
        dict(name="aw_table_6000", kind="aw_table", nk=6000, nant=64, nw=64, S=16, Q=16),
        # 32 w-planes of a wide field, most visibilities in few of them
        dict(name="wstack_4096", kind="wstack", N=4096, n=4000000, planes=32, S=8, Q=8),
        # the same field in sub-grids
        dict(name="wtowers_4096", kind="wtowers", N=4096, n=2000000, s=256, margin=16, winc=100.0,
             S=8, Q=8, wrange=500.0, wstep=10.0, npixff=64),
        # distributed FFT: four facets of the 8192^2 image, its 22 x 22 subgrids, and back
        dict(name="recombine_8192", kind="recombine", N=8192, spacing=128, yB=1280, yN=1536,
             yP=2048, xA=384, xM=512, xMxN=144, nf=2, ns=22),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["conv", "conv", "driver", "wproj", "wproj", "diff", "aw", "aw", "aw_cycle",
                       "aw_table", "wstack", "wtowers", "recombine"])
    if kind == "conv":
        fp64 = rng.random() < 0.2
        return dict(kind=kind, N=_log(rng, 256, 4096), n=_log(rng, 1000, 200000 if fp64 else 4000000),
                    S=rng.randint(3, 16), Q=rng.choice([2, 4, 7, 8, 16]), sep=rng.random() < 0.6,
                    precision="fp64" if fp64 else "fp32")
    if kind == "driver":
        return dict(kind=kind, N=_log(rng, 256, 2048), n=_log(rng, 2000, 500000),
                    S=rng.randint(4, 12), Q=rng.choice([4, 8]))
    if kind == "wproj":
        fp64 = rng.random() < 0.2
        return dict(kind=kind, N=_log(rng, 512, 4096), n=_log(rng, 5000, 100000 if fp64 else 3000000),
                    S=rng.randint(7, 16), Q=rng.choice([4, 8]), wrange=float(rng.randint(50, 500)),
                    wstep=float(rng.randint(8, 25)), npixff=rng.choice([32, 48, 64]),
                    precision="fp64" if fp64 else "fp32")
    if kind == "diff":
        return dict(kind=kind, N=rng.choice([512, 1024, 1500, 2048, 4096]), n=_log(rng, 20000, 2000000),
                    S=rng.randint(4, 12), Q=rng.choice([4, 8]))
    if kind in ("aw", "aw_cycle"):
        return dict(kind=kind, N=_log(rng, 1024, 8192) & ~1, nant=rng.randint(8, 48),
                    ntime=rng.randint(9, 99), nchan=rng.randint(5, 64), wbins=rng.choice([16, 32, 64]))
    if kind == "aw_table":
        return dict(kind=kind, nk=_log(rng, 50, 6000), nant=rng.randint(4, 64), nw=rng.randint(1, 64),
                    S=rng.choice([8, 16, 16, 16]), Q=rng.choice([4, 8, 16]))
    if kind == "wstack":
        return dict(kind=kind, N=rng.choice([1024, 1536, 2048, 4096]), n=_log(rng, 100000, 4000000),
                    planes=rng.randint(3, 24), S=rng.randint(5, 10), Q=rng.choice([4, 8]))
    if kind == "wtowers":
        return dict(kind=kind, N=rng.choice([1024, 2048, 4096]), n=_log(rng, 50000, 2000000),
                    s=rng.choice([128, 256]), margin=rng.choice([12, 16, 24]),
                    winc=float(rng.randint(60, 200)), S=rng.randint(6, 10), Q=8,
                    wrange=float(rng.randint(100, 500)), wstep=10.0, npixff=64)
    if rng.random() < 0.5:  # small image, transforms of 216 points (not a power of two)
        return dict(kind=kind, N=512, spacing=4, yB=128, yN=140, yP=216, xA=128, xM=256, xMxN=136,
                    nf=rng.randint(1, 4), ns=rng.randint(1, 4))
    return dict(kind=kind, N=8192, spacing=128, yB=1280, yN=1536, yP=2048, xA=384, xM=512, xMxN=144,
                nf=rng.randint(1, 2), ns=rng.randint(3, 22))


# ------------------------------------------------------------------ inputs

THETA = {"conv": 0.08, "driver": 0.08, "diff": 0.08, "wproj": 0.1, "wstack": 0.1, "wtowers": 0.1,
         "aw": 0.05, "aw_cycle": 0.05, "aw_table": 0.05}


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 2654435761 % (1 << 62) + 1)


def _rand(g, *shape):
    return torch.rand(shape, dtype=F64, device="cuda", generator=g)


def _point_sources(g, uvw, nsrc, half_width):
    """Visibilities of a few point sources: sum of f exp(-2 pi i (u l + v m + w (n - 1)))."""
    l, m = (2 * _rand(g, 2, nsrc) - 1) * half_width
    f = torch.randn(nsrc, dtype=F64, device="cuda", generator=g)
    lmn = torch.stack([l, m, torch.sqrt(1 - l * l - m * m) - 1])
    vis = torch.zeros(len(uvw), dtype=C128, device="cuda")
    for k in range(nsrc):
        turns = uvw @ lmn[:, k]
        vis += torch.polar(f[k].expand(len(uvw)), -2 * math.pi * (turns - torch.round(turns)))
    return vis.to(C64)


def _radial(g, n, lam, w):
    """uvw with a radial density of 1/r inside 0.45 lam."""
    r, phi = 0.45 * lam * _rand(g, n), 2 * math.pi * _rand(g, n)
    return torch.stack([r * torch.cos(phi), r * torch.sin(phi), w], dim=1).contiguous()


def _taper(N, S, Q):
    """The oversampled separable kernel [Q, S] of a Kaiser taper over an N-pixel field."""
    far = numpy.kaiser(N + 1, 8.0)[:N] if N % 2 == 0 else numpy.kaiser(N, 8.0)
    big = numpy.zeros(N * Q)
    big[N * Q // 2 - N // 2:N * Q // 2 - N // 2 + N] = far
    a = numpy.fft.fftshift(numpy.fft.fft(numpy.fft.ifftshift(big))) / N
    start = N * Q // 2 - Q * (S // 2)
    return numpy.array([a[start + f:start + f + Q * S:Q] for f in range(Q)])


def _kernel(case):
    k = _taper(case["N"], case["S"], case["Q"])
    return k if case.get("sep", True) else k[:, None, :, None] * k[None, :, None, :]


def _tracks(case, seed):
    """Earth-rotation tracks of antennas at random places, every channel of every
    baseline: uvw [n, 3], a1, a2 [n], the w step and the grid's width in wavelengths."""
    rng = numpy.random.default_rng(seed)
    nant, lam = case["nant"], case["N"] / THETA[case["kind"]]
    e, n_, up = rng.normal(0, 1500.0, nant), rng.normal(0, 1500.0, nant), rng.normal(0, 5.0, nant)
    lat, dec = math.radians(-27.0), math.radians(-45.0)
    c = math.pi / 2 - lat
    x, y, z = e, -up * math.sin(c) + n_ * math.cos(c), up * math.cos(c) + n_ * math.sin(c)
    ha = numpy.radians(numpy.linspace(-60.0, 60.0, case["ntime"]))[:, None]
    v0 = x * numpy.sin(ha) + y * numpy.cos(ha)
    pos = numpy.stack([x * numpy.cos(ha) - y * numpy.sin(ha),
                       z * math.cos(dec) + v0 * math.sin(dec),
                       z * math.sin(dec) - v0 * math.cos(dec)], axis=2)
    i1, i2 = numpy.triu_indices(nant, 1)
    bl = torch.from_numpy(pos[:, i2] - pos[:, i1]).cuda().reshape(-1, 3)
    freq = torch.linspace(1.0, 1.3, case["nchan"], dtype=F64, device="cuda")
    scale = 0.45 * lam / (1.3 * float(torch.hypot(bl[:, 0], bl[:, 1]).max())) * (1 - 1e-9)
    uvw = (bl[:, None, :] * (freq[:, None] * scale)).reshape(-1, 3).contiguous()
    a1, a2 = (torch.from_numpy(i.astype(numpy.int32)).cuda().repeat(case["ntime"])
              .repeat_interleave(case["nchan"]) for i in (i1, i2))
    wstep = float(math.ceil(float(uvw[:, 2].abs().max()) / (case["wbins"] / 2)))
    return uvw, a1, a2, wstep, lam


def _beams(g, nant, npix, theta):
    """Smooth complex far fields, one per antenna: a Gaussian under a low-order phase screen."""
    c = (torch.arange(npix, dtype=F64, device="cuda") - npix // 2) / npix * theta
    m, l = torch.meshgrid(c, c, indexing="ij")
    k = torch.randn(nant, 6, 1, 1, dtype=F64, device="cuda", generator=g)
    sig = theta / 3 * (1 + 0.1 * k[:, 5])
    ph = (k[:, 0] * l + k[:, 1] * m) / theta * 0.2 + \
        (k[:, 2] * l * l + k[:, 3] * m * m + k[:, 4] * l * m) / theta ** 2 * 0.3
    return torch.polar(torch.exp(-(l * l + m * m) / (2 * sig ** 2)), 2 * math.pi * ph)


def _aw_table_inputs(case, seed):
    g = _gen(seed)
    A = _crop_far(_beams(g, case["nant"], 32, 0.05), case["S"])
    W = _w_table(0.05, 30.0 * (torch.arange(case["nw"], dtype=F64, device="cuda")
                               - case["nw"] // 2), 32, case["S"], case["Q"])
    a1, a2 = (torch.randint(case["nant"], (case["nk"],), device="cuda", generator=g).int()
              for _ in range(2))
    wi = torch.randint(case["nw"], (case["nk"],), device="cuda", generator=g).int()
    return A, W, a1, a2, wi


def _facet_layout(case):
    fs = case["N"] // case["spacing"]
    nf, ns = -(-case["N"] // case["yB"]), -(-case["N"] // case["xA"])
    fo = [fs * round(j * case["N"] / nf / fs) for j in range(nf)]
    so = [case["spacing"] * round(i * case["N"] / ns / case["spacing"]) for i in range(ns)]
    return fo[:case["nf"]], so[:case["ns"]]


def _pswf(case):
    """A Kaiser window of the prolate function's width, centred at yN // 2."""
    c = math.pi * case["yN"] * (case["xM"] - case["xA"]) / (4.0 * case["N"])
    return numpy.kaiser(case["yN"] + 1, c)[:-1]


def _inputs(case, seed):
    """The case's inputs on the GPU, from the seed alone."""
    kind, g = case["kind"], _gen(seed)
    if kind == "aw_table":
        return dict(zip(("A", "W", "a1", "a2", "wi"), _aw_table_inputs(case, seed)))
    if kind == "recombine":
        fo, so = _facet_layout(case)
        shape = (len(fo), len(fo), case["yB"], case["yB"])
        return dict(facets=torch.randn(shape, dtype=C128, device="cuda", generator=g), fo=fo, so=so)
    if kind in ("aw", "aw_cycle"):
        uvw, a1, a2, wstep, lam = _tracks(case, seed)
        d = dict(uvw=uvw, a1=a1, a2=a2, wstep=wstep, lam=lam,
                 beams=_beams(g, case["nant"], 32, THETA[kind]),
                 vis=_point_sources(g, uvw, 8, THETA[kind] / 2))
        if kind == "aw_cycle":
            d["model"] = torch.randn((case["N"],) * 2, dtype=C64, device="cuda", generator=g)
        return d
    N, n, theta = case["N"], case["n"], THETA[kind]
    lam = N / theta
    d = dict(lam=lam)
    if kind == "wstack":
        # power-law plane counts in random order, w spread over each plane's width
        rng = numpy.random.default_rng(seed)
        p = (1.0 + numpy.arange(case["planes"])) ** -1.5
        p = p[rng.permutation(case["planes"])]
        edge = torch.from_numpy(numpy.cumsum(p / p.sum())).cuda()
        plane = torch.searchsorted(edge, _rand(g, n)).clamp_(max=case["planes"] - 1)
        step = 1600.0 / max(1, case["planes"] - 1)
        w = -800.0 + step * (plane + _rand(g, n) - 0.5)
        d["plane"] = plane.int().cpu().numpy()
    else:
        w = (2 * _rand(g, n) - 1) * case.get("wrange", 0.0)
    d["uvw"] = _radial(g, n, lam, w)
    d["vis"] = _point_sources(g, d["uvw"], 20, theta / 2)
    if kind in ("conv", "driver", "diff", "wstack"):
        d["kv"] = _kernel(case)
    if kind in ("conv", "wproj", "wtowers"):
        d["guv"] = torch.randn((N, N), dtype=C64, device="cuda", generator=g)
    if kind in ("driver", "diff"):
        d["image"] = torch.zeros((N, N), dtype=torch.float32, device="cuda")
        at = torch.randint(N // 4, 3 * N // 4, (2, 50), device="cuda", generator=g)
        d["image"][at[0], at[1]] = torch.randn(50, device="cuda", generator=g)
    return d


def prepare(case, seed):
    d = dict(_inputs(case, seed), case=case)
    kind = case["kind"]
    if kind in ("conv", "wproj") and case["precision"] == "fp64":
        d["vis"], d["guv"] = d["vis"].to(C128), d["guv"].to(C128)
    if kind == "driver":
        for k in ("uvw", "vis", "image"):
            d[k] = d[k].cpu().numpy()
        d["vis"] = d["vis"].astype(numpy.complex128)
    elif kind == "diff":
        table = engine.KernelTable.from_gcf(d["kv"], 0, C64)
        d["op"] = autograd.GriddingOperator(d["uvw"], d["lam"], (case["N"],) * 2, table)
        d["image"].requires_grad_(True)
    elif kind in ("aw", "aw_cycle"):
        d["op"] = awproj.AWProjection(THETA[kind], d["lam"], d["uvw"], d["a1"], d["a2"], d["beams"],
                                      d["wstep"], N=case["N"])
    elif kind == "recombine":
        d["rc"] = recombine.Recombine(*(case[k] for k in ("N", "spacing", "yB", "yN", "yP", "xA", "xM",
                                                          "xMxN")), pswf=_pswf(case))
    return d


# ------------------------------------------------------------------ the pass

def run(d):
    case, kind = d["case"], d["case"]["kind"]
    theta = THETA.get(kind)
    if kind == "conv":
        kw = dict(kv=d["kv"], precision=case["precision"])
        return (synthesis.conv_imaging(theta, d["lam"], d["uvw"], None, d["vis"], **kw),
                synthesis.conv_predict(theta, d["lam"], d["uvw"], None, d["guv"], **kw))
    if kind == "driver":
        return (*synthesis.do_imaging(theta, d["lam"], d["uvw"], None, d["vis"],
                                      synthesis.conv_imaging, kv=d["kv"]),
                synthesis.do_predict(theta, d["lam"], d["uvw"], None, d["image"],
                                     synthesis.conv_predict, kv=d["kv"]))
    if kind == "wproj":
        kw = dict(wstep=case["wstep"], NpixFF=case["npixff"], NpixKern=case["S"], Qpx=case["Q"],
                  precision=case["precision"])
        return (synthesis.w_cache_imaging(theta, d["lam"], d["uvw"], None, d["vis"], **kw),
                synthesis.w_cache_predict(theta, d["lam"], d["uvw"], None, d["guv"], **kw))
    if kind == "diff":
        v = d["op"].predict(d["image"])
        loss = (torch.abs(v - d["vis"]) ** 2).sum()
        return v.detach(), torch.autograd.grad(loss, d["image"])[0]
    if kind == "aw":
        d["op"].replan()
        grid = d["op"].grid(d["vis"])
        return grid, d["op"].degrid(grid)
    if kind == "aw_cycle":
        d["op"].replan()
        grid = torch.zeros_like(d["model"])
        return d["op"].degrid_grid(d["model"], d["vis"], grid, residual=True), grid
    if kind == "aw_table":
        return engine.aw_kernels(d["A"], d["W"], d["a1"], d["a2"], d["wi"])
    if kind == "wstack":
        return synthesis.w_stack_imaging(theta, d["lam"], d["uvw"], None, d["vis"], d["kv"],
                                         d["plane"])
    if kind == "wtowers":
        kw = dict(NpixFF=case["npixff"], NpixKern=case["S"], Qpx=case["Q"])
        args = (case["s"], case["margin"], case["winc"], case["wstep"])
        return (synthesis.w_towers_imaging(theta, d["lam"], d["uvw"], None, d["vis"], *args, **kw),
                synthesis.w_towers_predict(theta, d["lam"], d["uvw"], None, d["guv"], *args, **kw))
    subgrids = d["rc"].recombine(d["facets"], d["fo"], d["fo"], d["so"], d["so"])
    return subgrids, d["rc"].split(subgrids, d["so"], d["so"], d["fo"], d["fo"])


def work(case):
    kind = case["kind"]
    if kind == "recombine":
        nf, ns = case["nf"] ** 2, case["ns"] ** 2
        xy = case["xM"] * case["yP"] // case["N"]
        xn = case["xM"] * case["yN"] // case["N"]
        fft = lambda m, rows: 5.0 * m * math.log2(m) * rows  # noqa: E731
        one = fft(case["yP"], case["yB"] + case["ns"] * xn) + \
            fft(xy, case["ns"] * (case["yB"] + case["ns"] * xn))
        return {"bytes": 16.0 * (2 * nf * case["yB"] ** 2 + 2 * ns * case["xA"] ** 2),
                "flops": 2 * nf * one + 2 * ns * fft(case["xM"], 2 * case["xM"])}
    if kind == "aw_table":
        sub = case["nk"] * case["Q"] ** 2
        per = 6 * 1024 + 5 * 32 * 5 * (32 + case["S"])  # a 32 x 32 product and its pruned transform
        return {"bytes": 8.0 * sub * case["S"] ** 2 + 16.0 * case["nw"] * (case["Q"] * case["S"]) ** 2,
                "flops": float(sub * per)}
    N = case["N"]
    if kind in ("aw", "aw_cycle"):
        n, S = case["nant"] * (case["nant"] - 1) // 2 * case["ntime"] * case["nchan"], 16
        # uvw, key, visibility in and out, both grids, and the kernel slices: about one in three is new
        return {"bytes": n * (24.0 + 4 + 8 + 8) + 16.0 * N * N + n / 3 * 8.0 * S * S,
                "flops": 2 * 8.0 * n * S * S}
    n, S, wide = case["n"], case["S"], 2 if case.get("precision") == "fp64" else 1
    fft = 5.0 * N * N * 2 * math.log2(N)
    flops = 2 * 8.0 * n * S * S
    if kind == "wstack":
        return {"bytes": n * (24.0 + 4 + 8) + 8.0 * N * N * (1 + 2 * case["planes"]),
                "flops": flops / 2 + case["planes"] * (fft + 14.0 * N * N)}
    if kind == "driver":
        return {"bytes": n * (24.0 + 16 + 24 + 16) + 8.0 * N * N * 2 + 4.0 * N * N,
                "flops": 1.5 * flops + 3 * fft}
    if kind == "diff":
        return {"bytes": n * (24.0 + 8 + 8) + 8.0 * N * N, "flops": flops + 2 * fft}
    if kind == "wtowers":
        return {"bytes": n * (48.0 + 16) + 16.0 * N * N, "flops": flops + 4 * fft}
    return {"bytes": n * (24.0 + wide * 16) + wide * 16.0 * N * N, "flops": flops}


# ------------------------------------------------------------------ in 64 bits

def _centred(a, inverse, dims=(-2, -1)):
    f = torch.fft.ifftn if inverse else torch.fft.fftn
    return torch.fft.fftshift(f(torch.fft.ifftshift(a, dims), dim=dims), dims)


def _oversampled(far, S, Q):
    """Kernels [.., Q, Q, S, S] of square far fields [.., F, F]."""
    F = far.shape[-1]
    lo, M = F * Q // 2 - F // 2, F * Q
    big = torch.zeros(far.shape[:-2] + (M, M), dtype=C128, device="cuda")
    big[..., lo:lo + F, lo:lo + F] = far
    a = _centred(big, False)
    start = M // 2 - Q * (S // 2)
    a = a[..., start:start + Q * S, start:start + Q * S]
    a = a.reshape(far.shape[:-2] + (S, Q, S, Q))
    return a.movedim((-3, -1), (-4, -3)).contiguous()


def _crop_far(far, S):
    return _oversampled(far, S, 1)[..., 0, 0, :, :].contiguous()


def _pixels(N, theta):
    c = (torch.arange(N, dtype=F64, device="cuda") - N // 2) / N * theta
    return 1 - torch.sqrt(1.0 - c[None, :] ** 2 - c[:, None] ** 2)


def _turn(x):
    return torch.polar(torch.ones_like(x), 2 * math.pi * (x - torch.round(x)))


def _w_table(theta, w, npixff, S, Q):
    return torch.stack([_oversampled(_turn(-float(v) * _pixels(npixff, theta)), S, Q) for v in w])


def _aw_table(A, W, a1, a2, wi, S, Q):
    """(A1 conv A2) conv W of every key, 'same' crops, [nk, Q, Q, S, S]."""
    M, lo = 2 * S, (S - 1) // 2
    fA = torch.fft.fft2(A, s=(M, M))
    out = torch.empty((len(a1), Q, Q, S, S), dtype=C128, device="cuda")
    fW = torch.fft.fft2(W, s=(M, M))
    for k in range(0, len(a1), 256):
        i, j, w = (t[k:k + 256].long() for t in (a1, a2, wi))
        a = torch.fft.ifft2(fA[i] * fA[j])[:, lo:lo + S, lo:lo + S]
        a = torch.fft.fft2(a, s=(M, M))[:, None, None]
        out[k:k + 256] = torch.fft.ifft2(a * fW[w])[..., lo:lo + S, lo:lo + S]
    return out


def _cells(uv, lam, N, Q, S):
    """Footprint origin and fraction of coordinates along one axis."""
    f = torch.round(-(N // 2 + (uv / lam) * N) * Q).long()
    x = -torch.div(f, Q, rounding_mode="floor")
    return x - S // 2, f - torch.div(f, Q, rounding_mode="floor") * Q


class _Taps:
    """The taps of visibilities on a stack of N x N grids, one position in the footprint at a time."""

    def __init__(self, uvw, lam, N, kernels, Q, S, group=None, layer=None):
        x, xf = _cells(uvw[:, 0], lam, N, Q, S)
        y, yf = _cells(uvw[:, 1], lam, N, Q, S)
        self.base, self.N, self.S, self.kernels = y * N + x, N, S, kernels
        if layer is not None:
            self.base = self.base + layer * (N * N)
        self.row = (xf, yf)
        if kernels.dim() == 2:
            return
        self.kernels = kernels.reshape(-1, S * S)
        self.row = yf * Q + xf + (0 if group is None else group * (Q * Q))

    def each(self):
        for dy in range(self.S):
            for dx in range(self.S):
                if self.kernels.dim() == 2 and isinstance(self.row, tuple):
                    k = self.kernels[self.row[1], dy] * self.kernels[self.row[0], dx]
                else:
                    k = self.kernels[self.row, dy * self.S + dx]
                yield self.base + (dy * self.N + dx), k

    def grid(self, vis, layers=1):
        out = torch.zeros((layers * self.N * self.N, 2), dtype=F64, device="cuda")
        v = vis.to(C128)
        for at, k in self.each():
            out.index_add_(0, at, torch.view_as_real(k * v))
        out = torch.view_as_complex(out)
        return out.reshape((self.N, self.N) if layers == 1 else (layers, self.N, self.N))

    def degrid(self, grid):
        flat = grid.reshape(-1).to(C128)
        out = torch.zeros(len(self.base), dtype=C128, device="cuda")
        for at, k in self.each():
            out += flat[at] * k
        return out


def _w_groups(w, wstep):
    j = torch.round(w / wstep).long()
    lo, hi = int(j.min()), int(j.max())
    return j - lo, wstep * torch.arange(lo, hi + 1, dtype=F64, device="cuda")


def _exact_driver(case, d):
    N, lam, uvw, vis = case["N"], d["lam"], d["uvw"].clone(), d["vis"].to(C128).clone()
    flip = uvw[:, 1] < 0
    uvw[flip] = -uvw[flip]
    vis[flip] = torch.conj(vis[flip]).resolve_conj()
    x, y = _cells(uvw[:, 0], lam, N, 1, 0)[0], _cells(uvw[:, 1], lam, N, 1, 0)[0]
    cell = x * N + y
    weight = 1.0 / torch.bincount(cell, minlength=N * N)[cell].double()
    kv = torch.from_numpy(d["kv"]).cuda()
    taps = _Taps(uvw, lam, N, kv, case["Q"], case["S"])
    images = []
    for v in (vis * weight, weight):
        g = taps.grid(v)
        if N % 2 == 0:
            g[1:, 1:] += torch.conj(g[1:, 1:].flip(0, 1)).resolve_conj()
        else:
            g += torch.conj(g.flip(0, 1)).resolve_conj()
        images.append(_centred(g, True).real)
    top = float(images[1].max())
    taps = _Taps(d["uvw"], lam, N, kv, case["Q"], case["S"])
    out = taps.degrid(_centred(d["image"].to(C128), False))
    return (images[0] / top, images[1] / top, top, torch.view_as_real(out))


def _exact_towers(case, d):
    N, s, lam, theta = case["N"], case["s"], d["lam"], THETA["wtowers"]
    C, uvw = s - case["margin"], d["uvw"]
    ub, vb = (torch.floor(uvw[:, k] * theta / C).long() for k in (0, 1))
    wp = torch.round(uvw[:, 2] / case["winc"]).long()
    mid = lambda b: torch.div(C * b + C * (b + 1), 2, rounding_mode="floor")  # noqa: E731
    rel = torch.stack([uvw[:, 0] - mid(ub) / theta, uvw[:, 1] - mid(vb) / theta,
                       uvw[:, 2] - wp * case["winc"]], dim=1)
    span = lambda b: int(b.max() - b.min()) + 1  # noqa: E731
    chunk = (vb - vb.min()) * span(ub) + ub - ub.min()
    used, layer = torch.unique(chunk * span(wp) + wp - wp.min(), return_inverse=True)
    plane = (used % span(wp) + wp.min()).double() * case["winc"]
    chunks, of = torch.unique(torch.div(used, span(wp), rounding_mode="floor"), return_inverse=True)
    x0 = N // 2 + mid(chunks % span(ub) + ub.min()) - s // 2
    y0 = N // 2 + mid(torch.div(chunks, span(ub), rounding_mode="floor") + vb.min()) - s // 2
    group, w = _w_groups(rel[:, 2], case["wstep"])
    taps = _Taps(rel, s / theta, s, _w_table(theta, w, case["npixff"], case["S"], case["Q"]),
                 case["Q"], case["S"], group, layer)
    pix = _pixels(s, theta)
    stack = taps.grid(d["vis"], len(used)).reshape(-1, s, s)
    sub = torch.zeros((len(chunks), s, s), dtype=C128, device="cuda")
    for p in range(len(used)):
        sub[of[p]] += _centred(stack[p], True) * _turn(-plane[p] * pix)
    wide = torch.zeros((N + 2 * s, N + 2 * s), dtype=C128, device="cuda")  # cells outside fall off
    inner = wide[s:s + N, s:s + N]
    corners = list(zip(y0.tolist(), x0.tolist()))
    for c, (y, x) in enumerate(corners):
        wide[s + y:2 * s + y, s + x:2 * s + x] += _centred(sub[c], False)
    grid = inner.clone()
    inner.copy_(d["guv"])
    wide[:s] = wide[s + N:] = 0
    wide[:, :s] = wide[:, s + N:] = 0
    for p in range(len(used)):
        y, x = corners[int(of[p])]
        image = _centred(wide[s + y:2 * s + y, s + x:2 * s + x], True)
        stack[p] = _centred(image * _turn(-plane[p] * pix), False)
    return grid, taps.degrid(stack)


class _Facets:
    """The recombination's steps along an axis, centred arrays (last axis)."""

    def __init__(self, case):
        self.c = case
        N, yN, yP, xM = case["N"], case["yN"], case["yP"], case["xM"]
        self.xy, self.xn = xM * yP // N, xM * yN // N
        p = torch.from_numpy(_pswf(case)).cuda()
        self.Fb = 1 / self.mid(p, case["yB"])
        step = N // xM
        self.Fn = p[(yN // 2) % step::step]
        x = (torch.arange(yN, dtype=F64, device="cuda") - yN // 2) * (xM / N)
        m = p * torch.sinc(x)
        m[0] = 0  # the window is symmetric: its unpaired edge sample is left out
        self.m = self.xy * self.mid(self.fft(self.pad(m.to(C128), yP), True).real, case["xMxN"])
        self.fold = (case["xMxN"] - self.xy) // 2

    @staticmethod
    def mid(a, n):
        lo = a.shape[-1] // 2 - n // 2
        return a[..., lo:lo + n]

    @staticmethod
    def pad(a, n):
        out = torch.zeros(a.shape[:-1] + (n,), dtype=a.dtype, device="cuda")
        lo = n // 2 - a.shape[-1] // 2
        out[..., lo:lo + a.shape[-1]] = a
        return out

    @staticmethod
    def fft(a, inverse):
        return _centred(a, inverse, (-1,))

    def to_facet_image(self, a):
        return self.fft(self.pad(a * self.Fb, self.c["yP"]), True)

    def window(self, a, off):
        w = self.m * self.mid(torch.roll(a, -off * self.c["yP"] // self.c["N"], -1), self.c["xMxN"])
        s = self.mid(w, self.xy).clone()
        if self.fold:
            s[..., :self.fold] += w[..., -self.fold:]
            s[..., -self.fold:] += w[..., :self.fold]
        return self.Fn * self.mid(self.fft(s, False), self.xn)

    def unwindow(self, a, off):
        s = self.fft(self.pad(self.Fn * a, self.xy), True)
        w = self.pad(s, self.c["xMxN"])
        if self.fold:
            w[..., -self.fold:] = s[..., :self.fold]
            w[..., :self.fold] = s[..., -self.fold:]
        p = torch.roll(self.pad(self.m * w, self.c["yP"]), off * self.c["yP"] // self.c["N"], -1)
        return self.mid(self.fft(p, False), self.c["yB"])


def _exact_recombine(case, d):
    f, (fo, so) = _Facets(case), _facet_layout(case)
    xM, xn, N = case["xM"], f.xn, case["N"]
    sums = torch.zeros((len(so), len(so), xM, xM), dtype=C128, device="cuda")
    lo = xM // 2 - xn // 2
    part = torch.zeros((xM, xM), dtype=C128, device="cuda")
    shift = lambda o: o * xM // N  # noqa: E731
    for j0, o0 in enumerate(fo):
        for j1, o1 in enumerate(fo):
            rows = f.to_facet_image(d["facets"][j0, j1])
            for i1, s1 in enumerate(so):
                cols = f.to_facet_image(f.window(rows, s1).transpose(0, 1))
                for i0, s0 in enumerate(so):
                    part[lo:lo + xn, lo:lo + xn] = f.window(cols, s0).transpose(0, 1)
                    sums[i0, i1] += torch.roll(part, (shift(o0), shift(o1)), (0, 1))
    cut = xM // 2 - case["xA"] // 2
    for i in range(len(so)):
        sums[i] = _centred(sums[i], True)
    subgrids = sums[..., cut:cut + case["xA"], cut:cut + case["xA"]].contiguous()
    sums.zero_()
    sums[..., cut:cut + case["xA"], cut:cut + case["xA"]] = subgrids
    for i in range(len(so)):
        sums[i] = _centred(sums[i], False)
    facets = torch.zeros_like(d["facets"])
    for j0, o0 in enumerate(fo):
        for j1, o1 in enumerate(fo):
            for i0, s0 in enumerate(so):
                row = torch.zeros((xn, case["yB"]), dtype=C128, device="cuda")
                for i1, s1 in enumerate(so):
                    a = torch.roll(sums[i0, i1], (-shift(o0), -shift(o1)), (0, 1))
                    row += f.unwindow(a[lo:lo + xn, lo:lo + xn], s1)
                facets[j0, j1] += f.unwindow(row.transpose(0, 1), s0).transpose(0, 1)
            facets[j0, j1] *= f.Fb[:, None] * f.Fb
    return subgrids, facets


def exact(case, seed):
    kind, d = case["kind"], _inputs(case, seed)
    theta, N, S, Q = THETA.get(kind), case.get("N"), case.get("S", 16), case.get("Q", 16)
    if kind == "aw_table":
        return _aw_table(d["A"], d["W"], d["a1"], d["a2"], d["wi"], S, Q)
    if kind == "recombine":
        return _exact_recombine(case, d)
    if kind == "driver":
        out = _exact_driver(case, d)
        return (*out[:3], torch.view_as_complex(out[3]).cpu().numpy())
    if kind == "wtowers":
        return _exact_towers(case, d)
    if kind in ("aw", "aw_cycle"):
        group, w = _w_groups(d["uvw"][:, 2], d["wstep"])
        key = (d["a1"].long() * case["nant"] + d["a2"]) * len(w) + group
        used, row = torch.unique(key, return_inverse=True)
        pair = torch.div(used, len(w), rounding_mode="floor")
        table = _aw_table(_crop_far(d["beams"], S), _w_table(theta, w, 32, S, Q),
                          torch.div(pair, case["nant"], rounding_mode="floor"),
                          pair % case["nant"], used % len(w), S, Q)
        taps = _Taps(d["uvw"], d["lam"], N, table, Q, S, row)
        if kind == "aw":
            grid = taps.grid(d["vis"])
            return grid, taps.degrid(grid)
        v = taps.degrid(d["model"])
        return v, taps.grid(d["vis"] - v)
    if kind == "wproj":
        group, w = _w_groups(d["uvw"][:, 2], case["wstep"])
        taps = _Taps(d["uvw"], d["lam"], N, _w_table(theta, w, case["npixff"], S, Q), Q, S, group)
        return taps.grid(d["vis"]), taps.degrid(d["guv"])
    kv = torch.from_numpy(d["kv"]).cuda()
    if kind == "conv":
        taps = _Taps(d["uvw"], d["lam"], N, kv, Q, S)
        return taps.grid(d["vis"]), taps.degrid(d["guv"])
    if kind == "diff":
        taps = _Taps(d["uvw"], d["lam"], N, kv, Q, S)
        v = taps.degrid(_centred(d["image"].to(C128), False))
        taps.kernels = torch.conj(taps.kernels).resolve_conj()
        g = _centred(taps.grid(2 * (v - d["vis"].to(C128))), True).real * (N * N)
        return v, g
    image, pix = torch.zeros((N, N), dtype=C128, device="cuda"), _pixels(N, theta)
    plane = torch.from_numpy(d["plane"]).cuda()
    for p in range(int(plane.max()) + 1):
        sel = plane == p
        if bool(sel.any()):
            g = _Taps(d["uvw"][sel], d["lam"], N, kv, Q, S).grid(d["vis"][sel])
            image += _centred(g, True) * _turn(-d["uvw"][sel][:, 2].mean() * pix)
    return image
