"""Performance cases of the voxelwise T2map + T2part path.

Each case is a call (or a prepared batch's replay) that a program using this
package makes, through the package's public entry points: the device-pointer
C ABI for programs that keep volumes resident, the numpy functions for
programs that hold them on the host, and the prepared batch.  Images are
synthetic: three EPG decays per voxel (myelin, intra/extracellular, CSF) with
Rician noise and a share of background voxels below the threshold.
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.abspath("decaes.jl_gb300"))
import decaes_gb300 as D  # noqa: E402
from decaes_gb300 import _lib  # noqa: E402

SPWIN, MPWIN = (10e-3, 25e-3), (25e-3, 200e-3)
THRESHOLD = 200.0
MAPS = ("gdn", "ggm", "gva", "fnr", "snr", "alpha")
PARTS = ("sfr", "sgm", "mfr", "mgm")
# the most a drawn case may cost, in the unit of _cost (the largest listed case is the L-curve slab)
MOST = 0.6


def _case(call, X, m, TE, n, reg, K, precision, dtype, **kw):
    c = dict(call=call, x=X[0], y=X[1], z=X[2], nTE=m, TE=TE, nT2=n, T2lo=10e-3, reg=reg, nRefAngles=K,
             precision=precision, dtype=dtype, angle="search", RefConAngle=180.0, background=0.35, save=False)
    c.update(kw)
    return c


def listed():
    return [
        # a region of interest: the smallest call, latency and launches count
        dict(_case("host", (8, 8, 2), 32, 10e-3, 40, "chi2", 8, "fp64", "f64", background=0.0), name="roi_chi2_fp64"),
        # the reference's CPU-runnable configuration
        dict(_case("host", (32, 32, 4), 32, 10e-3, 40, "chi2", 8, "fp64", "f64", background=0.0), name="patch_chi2_fp64"),
        # a ragged strip resident on the device: less than two voxels a resident warp
        dict(_case("device", (61, 53, 1), 48, 10e-3, 40, "lcurve", 32, "mixed", "f32"), name="strip_lcurve48_mixed"),
        # one slice and a slab of the 48-echo volume of the benchmark
        dict(_case("device", (240, 240, 1), 48, 10e-3, 40, "lcurve", 32, "mixed", "f32"), name="slice_lcurve48_mixed"),
        dict(_case("device", (240, 240, 8), 48, 10e-3, 40, "lcurve", 32, "mixed", "f32"), name="slab_lcurve48_mixed"),
        # the same settings with the plain method (the default precision)
        dict(_case("device", (120, 120, 1), 48, 10e-3, 40, "lcurve", 32, "fp64", "f64"), name="slice_lcurve48_fp64"),
        # one slice of the 56-echo GCV volume
        dict(_case("device", (240, 240, 1), 56, 7e-3, 60, "gcv", 64, "mixed", "f32", T2lo=8e-3), name="slice_gcv56_mixed"),
        # the MATLAB toolbox's settings on a slab
        dict(_case("device", (240, 240, 4), 48, 10e-3, 40, "chi2", 8, "mixed", "f32"), name="slab_chi2k8_mixed"),
        # uneven volumes (24-64 echoes, three grids, chi2 and none) as one prepared batch
        dict(_case("batch", (64, 64, 2), 48, 9e-3, 48, "chi2", 32, "mixed", "f32", volumes=12), name="batch_uneven_mixed"),
        # a measured B1 map instead of the angle search, the discrepancy principle, a 150 degree control angle
        dict(_case("host", (61, 53, 7), 32, 10e-3, 40, "mdp", 32, "mixed", "f64", angle="b1", RefConAngle=150.0, save=True),
             name="b1_mdp_mixed"),
        # a fixed flip angle without regularization, every optional map saved
        dict(_case("host", (45, 37, 3), 32, 10e-3, 40, "none", 8, "fp64", "f64", angle="fixed", save=True),
             name="fixed_none_fp64"),
        # T2part alone on a saved distribution
        dict(_case("t2part", (240, 240, 16), 48, 10e-3, 40, "none", 32, "fp64", "f32"), name="slab_t2part"),
    ]


def _solves(c):
    """Least-squares solves of a voxel: those of the regularizer, and of the angle search."""
    s = {"none": 1, "chi2": 9, "mdp": 9, "lcurve": 27, "gcv": 16}[c["reg"]]
    return s + (min(c["nRefAngles"], 8) if c["angle"] == "search" else 0)


def _cost(c):
    """Seconds of a pass, roughly (what keeps a drawn case below the largest listed one)."""
    V = c["x"] * c["y"] * c["z"] * c.get("volumes", 1) * (1 - c["background"])
    if c["call"] == "t2part":
        return 1e-8 * V
    size = c["nTE"] * c["nT2"] / 1920.0
    s = 0.07 * _solves(c) * size ** 1.3
    if c["reg"] == "gcv":
        s *= 1.7
    if c["precision"] == "fp64":
        s *= 10 if c["reg"] == "gcv" else 6
    return 1e-6 * V * s


def draw(rng):
    while True:
        call = rng.choice(["device", "device", "device", "device", "host", "host", "batch", "t2part"])
        precision = rng.choice(["mixed", "mixed", "fp64"])
        reg = rng.choice(["lcurve", "lcurve", "chi2", "chi2", "gcv", "none", "mdp"])
        V = int(round(math.exp(rng.uniform(math.log(100), math.log(400000)))))
        z = rng.choice([1, 1, 2, 3, 5, 8])
        x = max(4, min(240, int(math.sqrt(V / z) * rng.uniform(0.7, 1.4))))
        y = max(4, min(240, V // (x * z)))
        m, n = rng.randint(24, 64), rng.choice([40, 48, 60, rng.randint(24, 60)])
        c = _case(call, (x, y, z), m, round(rng.uniform(5e-3, 12e-3), 5), n, reg, rng.choice([8, 16, 32, 64]), precision,
                  rng.choice(["f32", "f64"]), background=round(rng.uniform(0.3, 0.6), 2), save=rng.random() < 0.3,
                  RefConAngle=rng.choice([180.0, 180.0, 180.0, round(rng.uniform(140, 175), 1)]))
        if call == "host":
            c["angle"] = rng.choice(["search", "search", "b1", "fixed"])
        if call == "batch":
            c["volumes"], c["reg"], c["save"] = rng.randint(3, 12), "chi2", False
        if call == "t2part":
            c["precision"] = "fp64"
        if _cost(c) <= MOST:
            return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _epg(alpha, T2, m, TE, T1, beta):
    """CPMG echo amplitudes (len, m) of curves with refocusing angle alpha
    (degrees; control angle beta: the first pulse is alpha, later ones
    alpha/180 * beta) and relaxation time T2, by the extended phase graph:
    per half echo spacing relaxation and dephasing, then the pulse's rotation."""
    dt, dev = T2.dtype, T2.device
    rad = math.pi / 180
    e2 = torch.exp(-TE / 2 / T2)[:, None]
    e1 = math.exp(-TE / 2 / T1)
    F = torch.zeros(len(T2), m + 2, dtype=dt, device=dev)   # dephased states F_0, F_1, ...
    Fb = torch.zeros_like(F)                                # rephasing states F_-0, F_-1, ...
    Z = torch.zeros_like(F)
    F[:, 0] = Fb[:, 0] = torch.sin(alpha * rad / 2)
    out = torch.empty(len(T2), m, dtype=dt, device=dev)

    def half():
        nonlocal F, Fb, Z
        F, Fb, Z = F * e2, Fb * e2, Z * e1
        G = torch.roll(Fb, -1, 1)
        G[:, -1] = 0
        F = torch.roll(F, 1, 1)
        F[:, 0] = G[:, 0]
        Fb = G

    for i in range(m):
        half()
        a = (alpha if i == 0 else alpha / 180 * beta)[:, None] * rad
        c2, s2, s, co = torch.cos(a / 2) ** 2, torch.sin(a / 2) ** 2, torch.sin(a), torch.cos(a)
        F, Fb, Z = c2 * F + s2 * Fb + s * Z, s2 * F + c2 * Fb - s * Z, (s * (Fb - F)) / 2 + co * Z
        half()
        out[:, i] = Fb[:, 0].abs()
    return out


def _uniform(g, n, lo, hi):
    return lo + (hi - lo) * torch.rand(n, generator=g, device="cuda")


def _image(c, seed):
    """Echo trains (nTE, V) on the GPU, float32, and the voxels' refocusing angles."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    V, m = c["x"] * c["y"] * c["z"], c["nTE"]
    alpha = _uniform(g, V, 140.0, 180.0)
    if c["angle"] == "fixed":
        alpha = torch.full_like(alpha, 165.0)
    my, csf = _uniform(g, V, 0.05, 0.25), _uniform(g, V, 0.0, 0.05)
    t2 = (_uniform(g, V, 15e-3, 25e-3), _uniform(g, V, 60e-3, 90e-3), _uniform(g, V, 1.0, 2.0))
    amp, snr = _uniform(g, V, 500.0, 2000.0), _uniform(g, V, 50.0, 200.0)
    bg = torch.rand(V, generator=g, device="cuda") < c["background"]
    img = torch.empty(m, V, device="cuda")
    for a in range(0, V, 1 << 16):
        b = slice(a, min(V, a + (1 << 16)))
        s = sum((w * amp[b])[:, None] * _epg(alpha[b], t[b], m, c["TE"], 1.0, c["RefConAngle"])
                for w, t in zip((my[b], 1 - my[b] - csf[b], csf[b]), t2))
        s[bg[b]] = 0
        sigma = torch.where(bg, torch.full_like(amp, 8.0), amp / snr)[b][:, None]
        re, im = torch.randn(2, *s.shape, generator=g, device="cuda")
        img[:, b] = torch.hypot(s + sigma * re, sigma * im).T
    return img, alpha


def _options(c):
    kw = dict(MatrixSize=(c["x"], c["y"], c["z"]), nTE=c["nTE"], TE=c["TE"], nT2=c["nT2"], T2Range=(c["T2lo"], 2.0),
              Reg=c["reg"], nRefAngles=c["nRefAngles"], MinRefAngle=50.0, Threshold=THRESHOLD,
              RefConAngle=c["RefConAngle"], precision=c["precision"])
    if c["reg"] == "chi2":
        kw["Chi2Factor"] = 1.02
    if c["reg"] == "mdp":
        kw["NoiseLevel"] = 10.0
    if c["angle"] == "fixed":
        kw["SetFlipAngle"] = 165.0
    if c["save"]:
        kw.update(SaveResidualNorm=True, SaveDecayCurve=True, SaveRegParam=True)
    mo = D.T2mapOptions(**kw)
    return mo, D.T2partOptions.from_t2map(mo, SPWin=SPWIN, MPWin=MPWIN)


def _np_dtype(c):
    return np.float32 if c["dtype"] == "f32" else np.float64


def _dtype(c):
    return torch.float32 if c["dtype"] == "f32" else torch.float64


def _sizes(c):
    """Values of each output of T2map."""
    V = c["x"] * c["y"] * c["z"]
    n = {"dist": V * c["nT2"], **{k: V for k in MAPS}}
    if c["save"]:
        n.update(resnorm=V, decaycurve=V * c["nTE"], mu=V, chi2factor=V)
    return n


class _Resident:
    """A volume and its outputs on the device, and the C structs of its call."""

    def __init__(self, c, seed, new=None):
        self.mo, self.po = _options(c)
        dt = _dtype(c)
        self.code = _lib.F32 if c["dtype"] == "f32" else _lib.F64
        self.image = _image(c, seed)[0].to(dt).contiguous()
        new = new or (lambda key, n: torch.full((n,), math.nan, dtype=dt, device="cuda"))
        self.out = {k: new(k, n) for k, n in _sizes(c).items()}
        self.parts = {k: new(k, c["x"] * c["y"] * c["z"]) for k in PARTS}
        self.mc = _lib.T2mapOutC(**{k: t.data_ptr() for k, t in self.out.items()})
        self.pc = _lib.T2partOutC(**{k: t.data_ptr() for k, t in self.parts.items()})
        self.moc, self.poc = self.mo.to_c(), self.po.to_c()

    def volume(self):
        return _lib.VolumeC(mopts=self.moc, popts=self.poc, has_t2part=1, dtype=self.code,
                            d_image=self.image.data_ptr(), d_b1map=None, d_mout=self.mc, d_pout=self.pc)


class _Batch:
    """Resident volumes prepared once as a batch; each output is one tensor over all volumes."""

    def __init__(self, ctx, c, seed):
        cs = list(_batch_volumes(c))
        total = {k: sum(_sizes(v)[k] for v in cs) for k in _sizes(cs[0])}
        total.update({k: total["gdn"] for k in PARTS})
        self.out = {k: torch.full((n,), math.nan, dtype=_dtype(c), device="cuda") for k, n in total.items()}
        used = dict.fromkeys(total, 0)

        def part(key, n):
            used[key] += n
            return self.out[key][used[key] - n:used[key]]

        self.ctx, self.vols = ctx, [_Resident(v, seed * 64 + i, part) for i, v in enumerate(cs)]
        arr = (_lib.VolumeC * len(cs))(*[v.volume() for v in self.vols])
        torch.cuda.synchronize()
        self.h = ctx.L.decaes_batch_create(ctx.h, arr, len(cs))
        if not self.h:
            raise RuntimeError(ctx.L.decaes_last_error(ctx.h).decode())

    def __del__(self):
        if getattr(self, "h", None):
            self.ctx.L.decaes_batch_destroy(self.h)


def _batch_volumes(c):
    """The volumes of a batch: echo counts, grids, sizes and masks spread around the case's own."""
    r = np.random.default_rng(1000 * c["nTE"] + c["volumes"])
    for i in range(c["volumes"]):
        v = dict(c, nTE=int(r.integers(24, 65)), nT2=int(r.choice([40, 48, 60])), TE=float(r.uniform(5e-3, 12e-3)),
                 background=float(r.uniform(0.3, 0.6)), reg="chi2" if i % 2 == 0 else "none", call="device")
        v["x"], v["y"] = (max(4, int(c[k] * r.uniform(0.7, 1.7))) for k in "xy")
        yield v


def _stream():
    """The current torch stream for the C ABI (1 is the legacy default stream's handle, NULL the context's own stream)."""
    return C.c_void_p(torch.cuda.current_stream().cuda_stream or 1)


def _distribution(c, seed):
    """A distribution (x, y, z, nT2) as T2mapSEcorr saves it: a few spikes per voxel, NaN where it was not processed."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    V, n = c["x"] * c["y"] * c["z"], c["nT2"]
    d = torch.rand(n, V, generator=g, device="cuda") * 500
    d[torch.rand(n, V, generator=g, device="cuda") < 0.6] = 0
    d[:, torch.rand(V, generator=g, device="cuda") < c["background"]] = math.nan
    return d.to(_dtype(c))


def _host(t, *shape):
    """(echo or T2 bin, voxel) on the device -> a column-major array with the voxels' shape first."""
    return t.cpu().numpy().reshape(-1).reshape(shape, order="F")


def prepare(case, seed):
    c = case
    X = (c["x"], c["y"], c["z"])
    ctx = D.default_context()
    s = dict(case=c, ctx=ctx)
    if c["call"] == "device":
        s["vol"] = _Resident(c, seed)
    elif c["call"] == "batch":
        s["batch"] = _Batch(ctx, c, seed)
    elif c["call"] == "t2part":
        s["dist"] = _host(_distribution(c, seed), *X, c["nT2"])
        s["po"] = D.T2partOptions(MatrixSize=X, nT2=c["nT2"], T2Range=(c["T2lo"], 2.0), SPWin=SPWIN, MPWin=MPWIN)
    else:
        img, alpha = _image(c, seed)
        s["mo"], s["po"] = _options(c)
        s["image"] = np.asfortranarray(_host(img, *X, c["nTE"]), dtype=_np_dtype(c))
        s["b1"] = np.asfortranarray(_host(alpha, *X), dtype=_np_dtype(c)) if c["angle"] == "b1" else None
    return s


def run(state):
    s, ctx = state, state["ctx"]
    call = s["case"]["call"]
    if call == "device":
        v = s["vol"]
        ctx.check(ctx.L.decaes_t2map_t2part_device(ctx.h, C.byref(v.moc), C.byref(v.poc), C.c_void_p(v.image.data_ptr()),
                                                   v.code, None, C.byref(v.mc), C.byref(v.pc), _stream()))
        return [v.out, v.parts]
    if call == "batch":
        b = s["batch"]
        ctx.check(ctx.L.decaes_batch_run(b.h, _stream()))
        return b.out
    if call == "t2part":
        return D.T2partSEcorr(s["dist"], s["po"], ctx=ctx)
    maps, dist, parts = D.T2mapSEcorr_T2partSEcorr(s["image"], s["mo"], s["po"], b1map=s["b1"], ctx=ctx)
    return [{k: np.asarray(v) for k, v in maps.items()}, dist, parts]


def work(case):
    c = case
    vols = list(_batch_volumes(c)) if c["call"] == "batch" else [c]
    by = fl = 0.0
    e = 4 if c["dtype"] == "f32" else 8
    for v in vols:
        V = v["x"] * v["y"] * v["z"]
        if c["call"] == "t2part":
            by += e * V * (v["nT2"] + 4)
            fl += V * (1 - v["background"]) * 3.0 * v["nT2"]
            continue
        by += e * V * (v["nTE"] + v["nT2"] + 10 + ((3 + v["nTE"]) if v["save"] else 0))
        # the algorithm's FP64 operations of one solve at 48 x 40: Householder updates, or the Gram matrix's
        per = 1.7e5 if v["precision"] == "fp64" else 2.7e4
        fl += V * (1 - v["background"]) * per * _solves(v) * v["nTE"] * v["nT2"] / 1920.0
    return {"bytes": by, "flops": fl}


# ---------------------------------------------------------------------------
# values in 64 bits
# ---------------------------------------------------------------------------
def _nnls(A, b):
    """min ||A x - b||, x >= 0, by the active-set method of Lawson and Hanson."""
    n = A.shape[1]
    x, P = np.zeros(n), np.zeros(n, bool)
    for _ in range(10 * n):
        w = A.T @ (b - A @ x)
        w[P] = -1
        j = int(np.argmax(w))
        if w[j] <= 1e-13 * np.linalg.norm(b):
            break
        P[j] = True
        while True:
            z = np.zeros(n)
            z[P] = np.linalg.lstsq(A[:, P], b, rcond=None)[0]
            if z[P].min() > 0:
                break
            q = P & (z <= 0)
            x += (x[q] / (x[q] - z[q])).min() * (z - x)
            P &= x > 1e-14 * max(x.max(), 1e-300)
            x[~P] = 0
            if not P.any():
                z = x.copy()
                break
        x = z
    return x


def _t2_grid(c):
    return np.exp(np.linspace(math.log(c["T2lo"]), math.log(2.0), c["nT2"]))


def _exact_parts(d, t2):
    """T2part of distributions (V, nT2)."""
    win = lambda w: (t2 >= w[0] * (1 - 1e-9)) & (t2 <= w[1] * (1 + 1e-9))  # noqa: E731
    sp, mp, lt = win(SPWIN), win(MPWIN), np.log(t2)
    with np.errstate(invalid="ignore", divide="ignore"):
        tot, s, m = d.sum(1), d[:, sp].sum(1), d[:, mp].sum(1)
        nan = np.isnan(tot) | ~(tot > 0)
        return {"sfr": np.where(nan, np.nan, s / tot), "sgm": np.where(s > 0, np.exp(d[:, sp] @ lt[sp] / s), np.nan),
                "mfr": np.where(nan, np.nan, m / tot), "mgm": np.where(m > 0, np.exp(d[:, mp] @ lt[mp] / m), np.nan)}


def exact(case, seed):
    """T2part alone, and the unregularized fit at a fixed angle; the other
    cases' results are defined by the steps of their searches (a spline's
    minimum, a root to a tolerance, a curvature's corner), not by a value."""
    c = case
    X, V = (c["x"], c["y"], c["z"]), c["x"] * c["y"] * c["z"]
    t2 = _t2_grid(c)
    shaped = lambda p: {k: v.reshape(X, order="F") for k, v in p.items()}  # noqa: E731
    if c["call"] == "t2part":
        return shaped(_exact_parts(_distribution(c, seed).double().cpu().numpy().T, t2))
    if not (c["call"] == "host" and c["reg"] == "none" and c["angle"] == "fixed" and V <= 6000):
        return None
    img = _image(c, seed)[0].double().cpu().numpy().T  # (V, nTE)
    m, n = c["nTE"], c["nT2"]
    A = _epg(torch.full((n,), 165.0, dtype=torch.float64), torch.from_numpy(t2), m, c["TE"], 1.0,
             c["RefConAngle"]).numpy().T
    nan = lambda *s: np.full(s, np.nan)  # noqa: E731
    dist, fit = nan(V, n), nan(V, m)
    mx = img.max(1)
    for v in np.flatnonzero(img[:, 0] > THRESHOLD):
        dist[v] = _nnls(A, img[v] / mx[v]) * mx[v]
        fit[v] = A @ dist[v]
    res, lt, tot = fit - img, np.log(t2), dist.sum(1)
    with np.errstate(invalid="ignore", divide="ignore"):
        lg = dist @ lt / tot
        maps = {"gdn": tot, "ggm": np.exp(lg), "gva": np.expm1(((lt - lg[:, None]) ** 2 * dist).sum(1) / tot),
                "fnr": tot / np.sqrt((res ** 2).sum(1) / (m - 1)),
                "snr": mx / np.sqrt(((res - res.mean(1, keepdims=True)) ** 2).sum(1) / (m - 1)),
                "alpha": np.where(np.isnan(tot), np.nan, 165.0)}
    if c["save"]:
        maps.update(resnorm=np.sqrt((res ** 2).sum(1)))
    out = shaped(maps)
    out.update(echotimes=c["TE"] * np.arange(1, m + 1), t2times=t2, decaybasisset=A)
    if c["save"]:
        out["decaycurve"] = fit.reshape(*X, m, order="F")
    return [out, dist.reshape(*X, n, order="F"), shaped(_exact_parts(dist, t2))]
