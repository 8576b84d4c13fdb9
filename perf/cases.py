"""The calls whose speed this repository watches: imaging (ms2dirty) and
prediction (dirty2ms) through the public entry points, over the sizes, data
types and options that the configurations of ``cugridder_b200.synth``, the
benchmark and the tests use.

A case is a dict of plain values:

  entry   "plan"   ``Plan`` on device tensors (one channel, or ``nchan`` > 1)
          "batch"  ``Batch`` on device tensors: ``ndata`` uneven datasets
          "host"   ``curagridder.vis2dirty`` / ``dirty2vis`` on numpy arrays
          "nufft"  ``NufftPlan``: setpts and execute on device tensors
  way     "ms2dirty", "dirty2ms" or "cycle" (both, one after the other, as a
          major cycle of a deconvolution calls them); for nufft "type1", "type2"
  prec    "fp32" (uvw float64, the rest 32 bits) or "fp64"
  kernel  "es" or "learned" (the committed kernel of the width ``W``)

uvw follow the 4096 x 4096 configuration, scaled to each image: u, v normal
with sigma = ``sig`` x clip, clipped at 0.426 of the image's Nyquist limit, w
uniform within ``wfrac`` x clip; visibilities are complex N(0, 1), weights
U(0.5, 1.5).
"""
import math

import numpy as np
import torch

import cugridder_b200 as cg
from cugridder_b200.batch import Batch
from cugridder_b200.learn import load_kernel
from cugridder_b200.nufft import NufftPlan
from cugridder_b200.synth import BATCH_NYQUIST_FRACTION, C_LIGHT

REAL = {"fp32": torch.float32, "fp64": torch.float64}
CPLX = {"fp32": torch.complex64, "fp64": torch.complex128}


def _plan(name, **kw):
    c = dict(name=name, entry="plan", way="ms2dirty", nx=0, ny=0, fov=2.0, nrow=0, nchan=1, freq=1.5e8,
             prec="fp32", kernel="es", W=0, eps=1e-5, sig=0.3, wfrac=0.1, tuned=False)
    c.update(kw)
    return c


def listed():
    return [
        # the plain double-precision configuration, a major cycle on a small field
        _plan("cycle_256_fp64", way="cycle", nx=256, ny=256, nrow=100_000, freq=1.0e8, prec="fp64",
              wfrac=0.04),
        # a snapshot image of one short integration: the smallest call, where latency counts
        _plan("snapshot_512_fp32", nx=512, ny=512, nrow=20_000, eps=1e-4),
        # an image whose sides are neither equal nor powers of two
        _plan("image_1230x1002_fp32", nx=1230, ny=1002, fov=2.5, nrow=600_000),
        # prediction of a middle-sized field at the tighter single-precision accuracy
        _plan("predict_1500_fp32", way="dirty2ms", nx=1500, ny=1536, fov=3.0, nrow=3_000_000, eps=1e-6),
        # the kernel study's evaluation set with the learned kernel, plan defaults
        _plan("image_2048_learned", nx=2048, ny=2048, fov=3.0, nrow=10_000_000, kernel="learned", W=6,
              sig=0.25, wfrac=0.0625),
        # the headline workload, each direction, tuned in warm-up as the benchmark does
        _plan("image_4096_learned", nx=4096, ny=4096, fov=5.0, nrow=20_000_000, kernel="learned", W=6,
              tuned=True),
        _plan("predict_4096_learned", way="dirty2ms", nx=4096, ny=4096, fov=5.0, nrow=20_000_000,
              kernel="learned", W=6, tuned=True),
        # the double-precision leg at eps 1e-9 on the study's field
        _plan("cycle_2048_fp64_tight", way="cycle", nx=2048, ny=2048, fov=3.0, nrow=5_000_000,
              prec="fp64", eps=1e-9),
        # continuum imaging of several channels that share one uvw set
        _plan("channels_768_fp32", way="cycle", nx=768, ny=768, fov=2.0, nrow=200_000, nchan=6, eps=1e-4),
        # uneven datasets in one persistent launch per direction
        dict(name="batch_uneven_fp32", entry="batch", way="cycle", ndata=8, rows_lo=1e4, rows_hi=1e6,
             prec="fp32", kernel="learned", W=5, eps=1e-4),
        # the reference's numpy binding, drop-in calls on pageable host arrays
        _plan("host_1024_fp64", entry="host", way="cycle", nx=1024, ny=1024, nrow=500_000, freq=1.0e9,
              prec="fp64", eps=1e-6),
        # the generic front end
        dict(name="nufft_3d_type1_fp32", entry="nufft", way="type1", dim=3, n1=128, n2=128, n3=128,
             npts=2_000_000, prec="fp32", eps=1e-5),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    entry = rng.choice(["plan"] * 8 + ["batch", "host", "nufft"])
    prec = rng.choice(["fp32", "fp32", "fp64"])
    if entry == "nufft":
        dim = rng.choice([1, 2, 3])
        n = [2 * int(_log(rng, 16, {1: 200_000, 2: 600, 3: 70}[dim])) for _ in range(dim)] + [1] * (3 - dim)
        return dict(entry=entry, way=rng.choice(["type1", "type2"]), dim=dim, n1=n[0], n2=n[1], n3=n[2],
                    npts=int(_log(rng, 1e4, 2e6)), prec=prec,
                    eps=rng.choice([1e-3, 1e-4, 1e-5] if prec == "fp32" else [1e-5, 1e-7, 1e-9]))
    if entry == "batch":
        learned = prec == "fp32" and rng.random() < 0.5
        return dict(entry=entry, way="cycle", ndata=rng.randint(3, 10), rows_lo=1e4,
                    rows_hi=_log(rng, 1e5, 1e6), prec=prec, kernel="learned" if learned else "es",
                    W=5 if learned else 0, eps=1e-4)
    host = entry == "host"
    nx = 2 * int(_log(rng, 64, 512 if host else 2048))
    ny = nx if rng.random() < 0.6 else max(64, 2 * int(nx * rng.uniform(0.3, 0.7)))
    eps = rng.choice([1e-3, 1e-4, 1e-5, 1e-6] if prec == "fp32" else [1e-4, 1e-5, 1e-7, 1e-9])
    learned = prec == "fp32" and not host and eps in (1e-4, 1e-5) and rng.random() < 0.5
    nchan = 1 if host or rng.random() < 0.7 else rng.randint(2, 8)
    rows = _log(rng, 1e4, 1e6 if host else (2e7 if prec == "fp32" and nx < 3000 else 1e7))
    return _plan("", entry=entry, way=rng.choice(["ms2dirty", "dirty2ms", "cycle"]), nx=nx, ny=ny,
                 fov=round(rng.uniform(1.0, 5.0), 2), nrow=int(rows / nchan), nchan=nchan,
                 freq=1.0e8 * rng.randint(1, 10), prec=prec, kernel="learned" if learned else "es",
                 W={1e-4: 5, 1e-5: 6}[eps] if learned else 0, eps=eps,
                 sig=round(rng.uniform(0.15, 0.45), 3), wfrac=round(_log(rng, 0.02, 0.15), 4),
                 tuned=not host and rng.random() < 0.3)


# ---------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _uvw(g, nrow, nx, ny, fov, fmax, sig, wfrac):
    nyq = min(nx, ny) / (2 * math.radians(fov))  # wavelengths
    clip = BATCH_NYQUIST_FRACTION * nyq * C_LIGHT / fmax  # metres
    uvw = torch.empty((nrow, 3), dtype=torch.float64, device="cuda")
    uvw[:, :2] = (torch.randn((nrow, 2), generator=g, device="cuda", dtype=torch.float64)
                  * (sig * clip)).clamp_(-clip, clip)
    uvw[:, 2] = (torch.rand(nrow, generator=g, device="cuda", dtype=torch.float64) * 2 - 1) * (wfrac * clip)
    return uvw


def _complex(g, shape, prec):
    return torch.view_as_complex(torch.randn(tuple(shape) + (2,), generator=g, device="cuda", dtype=REAL[prec]))


def _freqs(case):
    n, f = case["nchan"], case["freq"]
    return [f] if n == 1 else [f * (1.0 + c / (n - 1)) for c in range(n)]


def _field(g, nrow, nchan, nx, ny, fov, freqs, sig, wfrac, prec):
    """One dataset on the device, and its image: noise for imaging, a model of
    random pixels for prediction."""
    shape = (nrow,) if nchan == 1 else (nrow, nchan)
    return dict(uvw=_uvw(g, nrow, nx, ny, fov, max(freqs), sig, wfrac), freqs=freqs, fov=fov,
                vis=_complex(g, shape, prec),
                wgt=torch.rand(shape, generator=g, device="cuda", dtype=REAL[prec]) + 0.5,
                model=_complex(g, (nx, ny), prec))


def _batch_specs(case, seed):
    """Dataset parameters as ``synth.batch_specs`` draws them, up to 1024 x 1024.
    Row counts, channels and sizes belong to the case, not to the seed."""
    import random

    r = random.Random(case["ndata"] * 7919)
    out = []
    for _ in range(case["ndata"]):
        nchan = r.randint(1, 16)
        freqs = [1.5e8] if nchan == 1 else [1.0e8 * (1.0 + c / (nchan - 1)) for c in range(nchan)]
        out.append(dict(nrow=max(100, int(_log(r, case["rows_lo"], case["rows_hi"]) / nchan)), nchan=nchan,
                        freqs=freqs, size=r.choice([512, 1024, 2048]), fov=round(r.uniform(1.0, 4.0), 2)))
    return out


def prepare(case, seed):
    g = _gen(seed)
    prec = case["prec"]
    if case["entry"] == "nufft":
        nm = (case["n1"], case["n2"], case["n3"])[:case["dim"]]
        pts = [(torch.rand(case["npts"], generator=g, device="cuda", dtype=torch.float64) * 2 - 1) * math.pi
               for _ in nm]
        c = _complex(g, (case["npts"],), prec)
        fk = _complex(g, tuple(reversed(nm)), prec)
        p = NufftPlan(1 if case["way"] == "type1" else 2, nm, iflag=1, eps=case["eps"], precision=prec)
        return dict(case=case, plan=p, pts=pts, c=c, fk=fk)
    if case["entry"] == "batch":
        data = []
        for s in _batch_specs(case, seed):
            d = _field(g, s["nrow"], s["nchan"], s["size"], s["size"], s["fov"], s["freqs"], 0.3, 0.1, prec)
            # each direction has buffers of its own, as a calibration loop keeps them
            d["image"], d["pred"] = torch.zeros_like(d["model"]), torch.zeros_like(d["vis"])
            data.append(d)
        batches = []
        for vis, img in (("vis", "image"), ("pred", "model")):
            b = Batch([dict(uvw=d["uvw"], freqs=d["freqs"], vis=d[vis], wgt=d["wgt"], dirty=d[img],
                            fov=d["fov"]) for d in data], epsilon=case["eps"], precision=prec)
            if case["kernel"] == "learned":
                k = load_kernel(case["W"])
                b.set_kernel("poly", k.W, k.horner)
            batches.append(b)
        return dict(case=case, data=data, image=batches[0], pred=batches[1])
    s = _field(g, case["nrow"], case["nchan"], case["nx"], case["ny"], case["fov"], _freqs(case),
               case["sig"], case["wfrac"], prec)
    s["case"] = case
    if case["entry"] == "host":
        # the reference's FP32 binding keeps uvw in 32 bits too
        r = np.float32 if prec == "fp32" else np.float64
        for k in ("uvw", "vis", "wgt", "model"):
            s[k] = s[k].cpu().numpy()
        s["uvw"], s["fov"] = s["uvw"].astype(r), float(r(s["fov"]))
        s["image"], s["pred"] = np.zeros_like(s["model"]), np.zeros_like(s["vis"])
        return s
    s["image"], s["pred"] = torch.zeros_like(s["model"]), torch.zeros_like(s["vis"])
    p = cg.Plan(case["nx"], case["ny"], case["fov"], case["eps"], precision=prec)
    if case["kernel"] == "learned":
        k = load_kernel(case["W"])
        p.set_kernel("poly", k.W, k.horner)
    if case["tuned"]:
        p.set_autotune(True)
    s["plan"] = p
    return s


# ---------------------------------------------------------------- one pass
def run(s):
    case = s["case"]
    way = case["way"]
    if case["entry"] == "nufft":
        s["plan"].setpts(*s["pts"])
        s["plan"].execute(s["c"], s["fk"])
        return s["fk"] if way == "type1" else s["c"]
    if case["entry"] == "batch":
        s["image"].ms2dirty()
        s["pred"].dirty2ms()
        return [[d["image"], d["pred"]] for d in s["data"]]
    out = []
    if case["entry"] == "host":
        f, fov, eps = s["freqs"], s["fov"], case["eps"]
        if case["prec"] == "fp64":
            if way != "dirty2ms":
                out.append(cg.vis2dirty(s["uvw"], f, s["vis"], s["wgt"], s["image"], fov, eps))
            if way != "ms2dirty":
                out.append(cg.dirty2vis(s["uvw"], f, s["pred"], s["wgt"], s["model"], fov, eps))
            return out
        n = s["uvw"].shape[0]
        if way != "dirty2ms":
            cg.ms2dirtyf_2(n, case["nx"], case["ny"], fov, f[0], s["uvw"], s["vis"], s["wgt"], s["image"],
                           eps, 2.0, 1)
            out.append(s["image"])
        if way != "ms2dirty":
            cg.dirty2msf_2(n, case["nx"], case["ny"], fov, f[0], s["uvw"], s["pred"], s["wgt"], s["model"],
                           eps, 2.0, 1)
            out.append(s["pred"])
        return out
    p, f = s["plan"], s["freqs"]
    if way != "dirty2ms":
        if case["nchan"] == 1:
            p.ms2dirty(s["uvw"], f[0], s["vis"], s["wgt"], s["image"])
        else:
            p.ms2dirty_chan(s["uvw"], f, s["vis"], s["wgt"], s["image"])
        out.append(s["image"])
    if way != "ms2dirty":
        if case["nchan"] == 1:
            p.dirty2ms(s["uvw"], f[0], s["model"], s["wgt"], s["pred"])
        else:
            p.dirty2ms_chan(s["uvw"], f, s["model"], s["wgt"], s["pred"])
        out.append(s["pred"])
    return out


# ---------------------------------------------------------------- what a pass cannot do without
def _width(case):
    return case["W"] or max(2, min(16, math.ceil(-math.log10(case["eps"] / 10.0))))


def _work_field(nrow, nchan, nx, ny, fov, W, prec, wfrac, ways):
    r = 4 if prec == "fp32" else 8
    n = nrow * nchan
    by = 24 * nrow + (2 * r + r) * n + 2 * r * nx * ny
    # w planes of the improved W-stacking (oversampling 2)
    clip = BATCH_NYQUIST_FRACTION * min(nx, ny) / (2 * math.radians(fov))
    half = math.radians(fov) / 2
    t = max(0.0, 1 - 2 * half * half)
    nw = max(2 * W, 2 * 2 * (1 - math.sqrt(t)) / 2 * max(1e-9, 2 * math.pi * wfrac * clip) / math.pi + W + 1)
    grid = 4.0 * nx * ny
    fl = 4.0 * W ** 3 * n + 5.0 * grid * math.log2(grid) * nw * 0.5 + 8.0 * nx * ny * nw
    return by * ways, fl * ways


def work(case):
    r = 4 if case["prec"] == "fp32" else 8
    if case["entry"] == "nufft":
        nk, W = case["n1"] * case["n2"] * case["n3"], _width(dict(case, W=0))
        g = nk * 2.0 ** case["dim"]
        return {"bytes": case["npts"] * (8 * case["dim"] + 2 * r) + 2 * r * nk,
                "flops": 4.0 * W ** case["dim"] * case["npts"] + 5.0 * g * math.log2(g)}
    ways = 2 if case["way"] == "cycle" else 1
    if case["entry"] == "batch":
        w = [_work_field(s["nrow"], s["nchan"], s["size"], s["size"], s["fov"], _width(case), case["prec"], 0.1, ways)
             for s in _batch_specs(case, 0)]
        return {"bytes": sum(x[0] for x in w), "flops": sum(x[1] for x in w)}
    b, f = _work_field(case["nrow"], case["nchan"], case["nx"], case["ny"], case["fov"], _width(case),
                       case["prec"], case["wfrac"], ways)
    return {"bytes": b, "flops": f}


def tolerance(case):
    # 32 bits: the same kernel and calls in 64 bits differ by 5e-7 (W = 5) to
    # 1.3e-6 (W = 7), sums in another order by 1e-7; 64 bits: sums in another
    # order differ by 8e-16, and another transform's rounding is of some 1e-15
    if case["prec"] == "fp32":
        return {"rel": 6e-6}
    return {"rel": 2e-14}


# ---------------------------------------------------------------- 64-bit sums
def _cheb(w, t, tol=1e-13):
    """exp(i w t) as sum_r A_r(w) B_r(t): Chebyshev interpolation in t."""
    t0, h = 0.5 * (t.min() + t.max()), max(0.5 * float(t.max() - t.min()), 1e-300)
    z = float(w.abs().max()) * h
    n = int(z * 1.3 + 24)
    nodes = torch.cos(math.pi * (torch.arange(n, device=t.device, dtype=torch.float64) + 0.5) / n)
    x = (t - t0) / h
    tx = [torch.ones_like(x), x]
    tn = [torch.ones_like(nodes), nodes]
    for _ in range(2, n):
        tx.append(2 * x * tx[-1] - tx[-2])
        tn.append(2 * nodes * tn[-1] - tn[-2])
    ph = torch.exp(1j * w[:, None] * (t0 + h * nodes)[None, :])
    A = [(ph @ tn[r].to(ph.dtype)) * ((1.0 if r == 0 else 2.0) / n) for r in range(n)]
    return A, tx[:n]


def _exact_field(d, freqs, nx, ny, sign, way, budget=8e11):
    uvw = torch.as_tensor(d["uvw"]).cuda().double()
    if float(nx) * ny * uvw.shape[0] * len(freqs) > budget:
        return None
    vis = torch.as_tensor(d["vis"]).cuda().to(torch.complex128).reshape(uvw.shape[0], -1)
    wgt = torch.as_tensor(d["wgt"]).cuda().double().reshape(uvw.shape[0], -1)
    model = torch.as_tensor(d["model"]).cuda().to(torch.complex128)
    pix = math.radians(d["fov"])
    l = (torch.arange(nx, device="cuda", dtype=torch.float64) - nx // 2) * (pix / nx)
    m = (torch.arange(ny, device="cuda", dtype=torch.float64) - ny // 2) * (pix / ny)
    r2 = l[:, None] ** 2 + m[None, :] ** 2
    n = torch.sqrt(1 - r2)
    t = -r2 / (1 + n)
    image = torch.zeros((nx, ny), device="cuda", dtype=torch.complex128)
    pred = torch.zeros_like(vis)
    for c, f in enumerate(freqs):
        k = 2 * math.pi * f / C_LIGHT
        for a in range(0, uvw.shape[0], 32768):
            u, v, w = (uvw[a:a + 32768, i] for i in range(3))
            A, B = _cheb(sign * k * w, t)
            U = torch.exp(1j * k * l[:, None] * u[None, :])
            V = torch.exp(1j * k * m[:, None] * v[None, :])
            q = vis[a:a + 32768, c] * wgt[a:a + 32768, c]
            p = torch.zeros_like(q)
            for Ar, Br in zip(A, B):
                if way != "dirty2ms":
                    image += Br * ((U * (q * Ar)) @ V.T)
                if way != "ms2dirty":
                    p += Ar.conj() * (U.conj() * ((model / n * Br) @ V.conj())).sum(0)
            pred[a:a + 32768, c] = p * wgt[a:a + 32768, c]
    out = []
    if way != "dirty2ms":
        out.append(image / n)
    if way != "ms2dirty":
        out.append(pred.reshape(tuple(d["vis"].shape)))
    return out


def exact(case, seed):
    s = prepare(case, seed)
    if case["entry"] == "nufft":
        nm = (case["n1"], case["n2"], case["n3"])[:case["dim"]]
        if float(case["npts"]) * case["n1"] * case["n2"] * case["n3"] > 6e12:
            return None
        type1 = case["way"] == "type1"
        c, fk = s["c"].to(torch.complex128), s["fk"].to(torch.complex128)
        ks = [torch.arange(n, device="cuda", dtype=torch.float64) - n // 2 for n in nm] + \
             [torch.zeros(1, device="cuda", dtype=torch.float64)] * (3 - len(nm))
        zero = torch.zeros_like(s["pts"][0])
        pts = s["pts"] + [zero] * (3 - len(nm))
        N1, N23 = case["n1"], case["n2"] * case["n3"]
        out = torch.zeros((N23, N1), device="cuda", dtype=torch.complex128)
        got = torch.zeros_like(c)
        step = max(64, min(16384, int(1e9 / 16 / max(N1, N23))))
        for a in range(0, case["npts"], step):
            e = [torch.exp(1j * k[:, None] * x[None, a:a + step]) for k, x in zip(ks, pts)]
            e23 = (e[2][:, None, :] * e[1][None, :, :]).reshape(N23, -1)
            if type1:
                out += (e23 * c[a:a + step]) @ e[0].T
            else:
                got[a:a + step] = (e23 * (fk.reshape(N23, N1) @ e[0])).sum(0)
        return out.reshape(tuple(reversed(nm))) if type1 else got
    if case["entry"] == "batch":
        out = []
        for spec, d in zip(_batch_specs(case, seed), s["data"]):
            r = _exact_field(d, spec["freqs"], spec["size"], spec["size"], -1, "cycle", budget=2.5e11)
            out.append([None, None] if r is None else r)
        return out if any(r[0] is not None for r in out) else None
    # the host binding's vis2dirty / dirty2vis use sign +1, plans the default -1
    return _exact_field(s, s["freqs"], case["nx"], case["ny"], 1 if case["entry"] == "host" else -1, case["way"])
