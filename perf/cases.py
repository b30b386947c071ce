"""The calls whose speed is measured: what each stands for, its inputs, one pass
through the public entry points, the work it cannot do without, and the values
a 64-bit evaluation gives.

A case is a dict of plain values.  ``path`` names the entry point:

  tabbed     TabbedBeamformer(...)(rf): delay tables of plane waves on a linear array
  dmas       TabbedDMASBeamformer with a short list of receive lags
  synthetic  SyntheticBeamformer: delays computed from synthetic points
  slsc       SyntheticSLSCBeamformer: short-lag spatial coherence
  matrix     SyntheticBeamformer in 3-D, diverging waves from a matrix array
  grad       TabbedBeamformer.differentiable, backward to data and delay tables
  grad_slow  SyntheticBeamformer.differentiable, backward to data and slowness
  batch      BatchBeamformer over uneven frames of both kinds
  bmode      Demodulator.bmode: envelope, percentile, log compression
"""
import math
import random

import numpy as np
import torch

import pycbf_gb300 as pg
from pycbf_gb300.batch import BatchBeamformer, BatchConfig
from pycbf_gb300.demod import Demodulator

C0 = 1540.0
FNUM = 1.5
THRESH = 1e-2
WINDOW_S = 64e-6      # record length of the frames of a batch
BATCH_NTX, BATCH_NRX, BATCH_NT = (1, 5, 11, 31, 75), (64, 128, 192), (1024, 2048, 4096)
BATCH_NX, BATCH_NZ = (128, 256, 512), (128, 256, 512, 1024)
DTYPES = {"float32": torch.float32, "float16": torch.float16, "bfloat16": torch.bfloat16,
          "int16": torch.int16}


def _linear(path, name=None, **kw):
    """A case on a linear array: 128 elements at 0.3 mm, 25 MHz, 256 x 512 pixels over
    38 x 40 mm from 5 mm depth, unless said otherwise."""
    case = dict(path=path, ntx=11, nrx=128, nt=2048, nx=256, nz=512, frames=1, fs=25e6,
                pitch=0.3e-3, width=38e-3, depth=40e-3, deg=10.0, data="float32",
                interp="cubic", sumtype="tx_and_rx")
    case.update(kw)
    if name:
        case["name"] = name
    return case


def _matrix(name=None, **kw):
    """A case on a matrix array: 32 x 32 elements at 0.3 mm, virtual sources on a 5 x 5
    grid 10 mm behind it, 20 MHz, voxels of 0.156 x 0.156 x 0.234 mm."""
    case = dict(path="matrix", side=32, sources=5, nt=2048, nx=64, ny=64, nz=128, frames=8,
                fs=20e6, pitch=0.3e-3, voxel=0.156e-3, voxel_z=0.234e-3, data="float16",
                interp="cubic", sumtype="tx_and_rx")
    case.update(kw)
    if name:
        case["name"] = name
    return case


def listed():
    return [
        # the ordinary frame: 11 plane waves on a 128-element array, a whole image
        _linear("tabbed", "tabbed_frame"),
        # the smallest call: one plane wave, a preview-sized image; launches count
        _linear("tabbed", "tabbed_preview", ntx=1, nrx=64, nt=1024, nx=64, nz=128),
        # a sequence of frames in half storage, beamformed in one call
        _linear("tabbed", "tabbed_8_frames_f16", frames=8, data="float16"),
        # converter counts from an acquisition system, two-point interpolation,
        # no size a multiple of anything
        _linear("tabbed", "tabbed_linear_i16_odd", ntx=7, nrx=97, nt=1999, nx=251, nz=509,
                interp="linear", data="int16"),
        # delay-multiply-and-sum over five receive lags
        _linear("dmas", "dmas_5_lags", lags=5, dmastype="ssr"),
        # many plane waves as far virtual sources on a 192-element array: one large image
        _linear("synthetic", "synthetic_frame", ntx=75, nrx=192, nt=4096, nx=512, nz=1024,
                fs=31.25e6, pitch=0.2e-3, width=38.4e-3, deg=18.0),
        # coherence image: per-element images, lags 1..16, axial kernel of 7 pixels
        _linear("slsc", "slsc_frame", ntx=31, nt=2048, fs=31.25e6, width=25.6e-3, pitch=0.2e-3,
                deg=16.0, nlag=16, nkern=3),
        # volume imaging: 25 diverging waves, 1024 elements, a run of volumes in half storage
        _matrix("matrix_8_volumes_f16"),
        # one training step: image, then gradients of the data and of both delay tables
        _linear("grad", "tabbed_gradients"),
        # one step of speed-of-sound estimation: per-element images, then gradients of
        # the data and of the slowness of every pixel
        _linear("grad_slow", "slowness_gradients", sumtype="tx_only"),
        # frames of many sizes, both kinds, in one replay
        dict(path="batch", name="batch_12_uneven", frames=12, sizes=64, data="float32"),
        # what follows every image: envelope, 99th percentile, decibels
        dict(path="bmode", name="bmode_frame", nx=256, nz=512, images=1, kmin=1e6, kmax=9e6,
             ks=25e6),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(("tabbed", "tabbed", "tabbed", "dmas", "synthetic", "synthetic", "slsc",
                       "matrix", "grad", "grad_slow", "batch", "bmode"))
    if path == "matrix":
        side, sources = rng.randint(8, 32), rng.randint(2, 5)
        case = _matrix(side=side, sources=sources, nt=rng.randint(1024, 2048),
                       frames=rng.randint(1, 8), nx=rng.randint(16, 64), ny=rng.randint(16, 64),
                       nz=_log(rng, 32, 128), data=rng.choice(("float32", "float16", "bfloat16")))
        return case
    if path == "batch":
        return dict(path="batch", frames=rng.randint(3, 12), sizes=rng.randrange(1 << 20),
                    data=rng.choice(("float32", "float16", "bfloat16")))
    if path == "bmode":
        return dict(path="bmode", nx=_log(rng, 32, 512), nz=_log(rng, 128, 1024),
                    images=rng.choice((1, 1, 3)), kmin=1e6, kmax=rng.choice((9e6, 6e6)), ks=25e6)
    case = _linear(path, ntx=_log(rng, 1, 75 if path in ("tabbed", "synthetic", "slsc") else 31),
                   nrx=_log(rng, 32, 192), nt=_log(rng, 512, 4096), nx=_log(rng, 32, 512),
                   nz=_log(rng, 64, 1024), deg=round(rng.uniform(5.0, 18.0), 1))
    # the records reach the deepest pixels, with something cut off now and then
    reach = rng.uniform(0.9, 1.3)
    case["fs"] = round(case["nt"] / (reach * WINDOW_S), 0)
    case["pitch"] = round(38.4e-3 / case["nrx"], 7)
    if path == "tabbed":
        case["interp"] = rng.choice(("cubic", "cubic", "cubic", "linear", "nearest"))
        case["data"] = rng.choice(("float32", "float32", "float16", "bfloat16", "int16"))
        case["sumtype"] = rng.choice(("tx_and_rx", "tx_and_rx", "tx_and_rx", "tx_only", "rx_only"))
        case["frames"] = rng.choice((1, 1, 1, 2, 3, 8))
    elif path == "synthetic":
        case["data"] = rng.choice(("float32", "float32", "float16", "bfloat16"))
        case["sumtype"] = rng.choice(("tx_and_rx", "tx_and_rx", "tx_only"))
        case["frames"] = rng.choice((1, 1, 2, 3))
    elif path == "dmas":
        case.update(lags=rng.randint(1, 10), dmastype=rng.choice(("ssr", "power")))
    elif path == "slsc":
        case.update(nlag=rng.randint(5, 16), nkern=rng.randint(1, 3))
    elif path in ("grad", "grad_slow"):
        case["ntx"] = min(case["ntx"], 16)
        case["sumtype"] = rng.choice(("tx_and_rx", "tx_only"))
    # no drawn case costs more than the largest listed one
    while _slots(case) > 8e9 or case["nrx"] * case["nx"] * case["nz"] * case["frames"] > 2e8:
        case["nx"], case["nz"] = max(32, case["nx"] * 2 // 3), max(64, case["nz"] * 2 // 3)
        case["frames"] = 1
    return case


def _slots(case):
    """(pixel, transmit, receive) triples of one pass."""
    if case["path"] == "matrix":
        return (case["nx"] * case["ny"] * case["nz"] * case["side"] ** 2 * case["sources"] ** 2
                * case["frames"])
    return case["nx"] * case["nz"] * case["ntx"] * case["nrx"] * case["frames"]


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _channels(shape, data, gen):
    """Band-limited echo-like channel data: white noise through a pulse of about five
    samples a cycle, strongest near the surface, in the type the acquisition delivers."""
    w = torch.randn(shape, generator=gen, device="cuda")
    k = torch.arange(-7, 8, device="cuda", dtype=torch.float32)
    h = (torch.exp(-0.5 * (k / 2.5) ** 2) * torch.cos(2 * math.pi * k / 5.0)).tolist()
    out = torch.zeros_like(w)
    nt = shape[-1]
    for m, c in enumerate(h):
        s = m - 7
        a, b = max(0, -s), min(nt, nt - s)
        out[..., a:b].add_(w[..., a + s:b + s], alpha=c)
    out.mul_(torch.exp(-torch.linspace(0.0, 1.5, nt, device="cuda")))
    if data == "int16":
        return (out * 2000.0).round().clamp(-32767, 32767).to(torch.int16)
    return out.to(DTYPES[data])


def _axes(case):
    xe = case["pitch"] * (np.arange(case["nrx"]) - (case["nrx"] - 1) / 2.0)
    th = np.radians(np.linspace(-case["deg"], case["deg"], case["ntx"])) if case["ntx"] > 1 \
        else np.zeros(1)
    x = np.linspace(-0.5 * case["width"], 0.5 * case["width"], case["nx"])
    z = np.linspace(5e-3, 5e-3 + case["depth"], case["nz"])
    return xe, th, x, z


def _tables(case):
    """tautx, apodtx, taurx, apodrx of plane waves (float32 on the GPU): ones on
    transmit, a Hann window inside the f-number mask on receive."""
    xe, th, x, z = (torch.as_tensor(v, device="cuda") for v in _axes(case))
    X, Z = (v.reshape(-1) for v in torch.meshgrid(x, z, indexing="ij"))
    origin = torch.where(th <= 0, xe[-1], xe[0])
    tautx = ((X - origin[:, None]) * torch.sin(th)[:, None] + Z * torch.cos(th)[:, None]) / C0
    dx = X - xe[:, None]
    taurx = torch.sqrt(dx * dx + Z * Z) / C0
    half = Z / (2 * FNUM)
    w = torch.cos(0.5 * math.pi * torch.clamp(dx / half, -1.0, 1.0)) ** 2
    apodrx = torch.where(dx.abs() < half, w, torch.zeros_like(w))
    f32 = lambda t: t.to(torch.float32).contiguous()  # noqa: E731
    return f32(tautx), torch.ones_like(f32(tautx)), f32(taurx), f32(apodrx)


def _geometry(case):
    """Synthetic-point arguments: plane waves as sources 10 m behind the array ('synthetic',
    'slsc' and batches), true plane waves ('grad_slow'), diverging waves in 3-D ('matrix')."""
    if case["path"] == "matrix":
        n, p = case["side"], case["pitch"]
        e = p * (np.arange(n) - (n - 1) / 2.0)
        ex, ey = (v.ravel() for v in np.meshgrid(e, e, indexing="ij"))
        s = np.linspace(-0.5 * n * p, 0.5 * n * p, case["sources"])
        sx, sy = (v.ravel() for v in np.meshgrid(s, s, indexing="ij"))
        nrx, ntx, back = n * n, len(sx), 10e-3
        axes = [case["voxel"] * (np.arange(m) - (m - 1) / 2.0) for m in (case["nx"], case["ny"])]
        axes.append(8e-3 + case["voxel_z"] * np.arange(case["nz"]))
        up = np.array([0.0, 0.0, 1.0])
        return dict(ovectx=np.stack([sx, sy, np.full(ntx, -back)], 1), nvectx=np.tile(up, (ntx, 1)),
                    doftx=np.zeros(ntx), alatx=np.full(ntx, math.atan2(n * p, back)),
                    t0tx=np.full(ntx, -back / C0), ovecrx=np.stack([ex, ey, np.zeros(nrx)], 1),
                    nvecrx=np.tile(up, (nrx, 1)), alarx=np.full(nrx, math.atan2(0.5, FNUM)), c0=C0,
                    pnts=np.stack([v.ravel() for v in np.meshgrid(*axes, indexing="ij")], 1))
    xe, th, x, z = _axes(case)
    origin = np.stack([np.where(th <= 0, xe[-1], xe[0]), np.zeros_like(th)], 1)
    nv = np.stack([np.sin(th), np.cos(th)], 1)
    zero = np.zeros(len(th))
    if case["path"] == "grad_slow":
        ov, t0, ala = origin, zero, zero
    else:
        ov = -10.0 * nv
        t0 = np.sum(nv * (ov - origin), -1) / C0
        d = origin - ov
        ala = np.arccos(np.abs(np.sum(d * nv, -1)) / np.linalg.norm(d, axis=-1))
    n = len(xe)
    return dict(ovectx=ov, nvectx=nv, doftx=zero.copy(), alatx=ala, t0tx=t0,
                ovecrx=np.stack([xe, np.zeros(n)], 1),
                nvecrx=np.stack([np.zeros(n), np.ones(n)], 1),
                alarx=np.full(n, math.atan2(0.5, FNUM)), c0=C0,
                pnts=np.stack([v.ravel() for v in np.meshgrid(x, z, indexing="ij")], 1))


def _counts(case):
    if case["path"] == "matrix":
        return case["sources"] ** 2, case["side"] ** 2, case["nx"] * case["ny"] * case["nz"]
    return case["ntx"], case["nrx"], case["nx"] * case["nz"]


def _rf_shape(case):
    ntx, nrx, _ = _counts(case)
    core = (ntx, nrx, case["nt"])
    return core if case["frames"] == 1 else (case["frames"],) + core


def _batch_frames(case):
    """The frames of a batch as cases of their own, sizes drawn from case['sizes']."""
    r = random.Random(case["sizes"])
    out = []
    for _ in range(case["frames"]):
        nrx, nt = r.choice(BATCH_NRX), r.choice(BATCH_NT)
        out.append(_linear(r.choice(("tabbed", "synthetic")), ntx=r.choice(BATCH_NTX), nrx=nrx,
                           nt=nt, nx=r.choice(BATCH_NX), nz=r.choice(BATCH_NZ), fs=nt / WINDOW_S,
                           pitch=0.2e-3, width=nrx * 0.2e-3, deg=16.0, data=case["data"]))
    return out


def _beamformer(case, tables=None):
    storage = "float32" if case["data"] == "int16" else case["data"]
    kw = dict(t0=0.0, dt=1.0 / case["fs"], nt=case["nt"], interp={"kind": case["interp"]},
              storage=storage)
    if case["path"] in ("tabbed", "dmas", "grad"):
        ttx, atx, trx, arx = _tables(case) if tables is None else tables
        kw.update(tautx=ttx, apodtx=atx, taurx=trx, apodrx=arx)
        if case["path"] == "dmas":
            return pg.TabbedDMASBeamformer(lags=list(range(1, case["lags"] + 1)),
                                           dmastype=case["dmastype"], **kw)
        return pg.TabbedBeamformer(sumtype=case["sumtype"], **kw)
    kw.update(_geometry(case))
    if case["path"] == "slsc":
        return pg.SyntheticSLSCBeamformer(grid_shape=(case["nx"], case["nz"]), nlag=case["nlag"],
                                          nkern=case["nkern"], **kw)
    return pg.SyntheticBeamformer(sumtype=case["sumtype"], **kw)


def _seeded(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _slowness(case, gen):
    """About 1/1540 s/m, smoothly different over the pixels by a few percent."""
    coarse = torch.randn((1, 1, 5, 9), generator=gen, device="cuda") * 0.01
    up = torch.nn.functional.interpolate(coarse, size=(case["nx"], case["nz"]), mode="bilinear",
                                         align_corners=True).reshape(-1)
    return ((1.0 + up) / C0).contiguous()


def _image_lines(case, gen):
    shape = (case["images"], case["nx"], case["nz"]) if case["images"] > 1 else \
        (case["nx"], case["nz"])
    return _channels(shape, "float32", gen) * 300.0


def _grad_shape(case):
    return (case["nrx"], case["nx"] * case["nz"]) if case["sumtype"] == "tx_only" else \
        (case["nx"] * case["nz"],)


def prepare(case, seed):
    gen = _seeded(seed)
    st = {"case": case}
    if case["path"] == "bmode":
        st["x"] = _image_lines(case, gen)
        st["demod"] = Demodulator(case["nz"], case["kmin"], case["kmax"], case["ks"])
        return st
    if case["path"] == "batch":
        frames = _batch_frames(case)
        st["rf"] = [_channels(_rf_shape(f), f["data"], gen) for f in frames]
        st["bf"] = BatchBeamformer([_beamformer(f) for f in frames],
                                   config=BatchConfig(branches=8))
        return st
    st["rf"] = _channels(_rf_shape(case), case["data"], gen)
    if case["path"] == "grad":
        st["tables"] = _tables(case)
        st["bf"] = _beamformer(case, st["tables"])
        st["gout"] = torch.randn(_grad_shape(case), generator=gen, device="cuda")
    elif case["path"] == "grad_slow":
        st["bf"] = _beamformer(case)
        st["slow"] = _slowness(case, gen)
        st["gout"] = torch.randn(_grad_shape(case), generator=gen, device="cuda")
    else:
        st["bf"] = _beamformer(case)
    return st


def run(state):
    path = state["case"]["path"]
    if path == "bmode":
        nd = 2 if state["x"].ndim == 3 else None
        return state["demod"].bmode(state["x"], image_ndim=nd)
    if path == "batch":
        return state["bf"](state["rf"])
    if path == "grad":
        rf = state["rf"].detach().requires_grad_(True)
        ttx = state["tables"][0].detach().requires_grad_(True)
        trx = state["tables"][2].detach().requires_grad_(True)
        img = state["bf"].differentiable(rf, tautx=ttx, taurx=trx)
        img.backward(state["gout"])
        return {"image": img.detach(), "rf": rf.grad, "tautx": ttx.grad, "taurx": trx.grad}
    if path == "grad_slow":
        rf = state["rf"].detach().requires_grad_(True)
        s = state["slow"].detach().requires_grad_(True)
        img = state["bf"].differentiable(rf, slowness=s)
        img.backward(state["gout"])
        return {"image": img.detach(), "rf": rf.grad, "slowness": s.grad}
    return state["bf"](state["rf"], out_as_numpy=False)


# ---------------------------------------------------------------------------
# the work of one pass
# ---------------------------------------------------------------------------
def _live_share(case):
    """Share of (receive, pixel) pairs inside the f-number mask, on a coarse grid."""
    if case["path"] == "matrix":
        n = case["side"]
        e = case["pitch"] * (np.arange(n) - (n - 1) / 2.0)
        x = case["voxel"] * (np.linspace(0, case["nx"] - 1, 9) - (case["nx"] - 1) / 2.0)
        z = 8e-3 + case["voxel_z"] * np.linspace(0, case["nz"] - 1, 17)
        d2 = (x[:, None] - e[None]) ** 2
        r2 = d2[:, None, :, None, None] + d2[None, :, None, :, None]
        return float(np.mean(r2 < (z / (2 * FNUM)) ** 2))
    xe, _, x, z = _axes(dict(case, nx=33, nz=65))
    return float(np.mean(np.abs(x[:, None, None] - xe[None, :, None]) < z / (2 * FNUM)))


def work(case):
    if case["path"] == "bmode":
        lo, hi = (int(np.argmin(np.abs(np.fft.rfftfreq(case["nz"], 1 / case["ks"]) - k)))
                  for k in (case["kmin"], case["kmax"]))
        m, lines = hi + 1 - lo, case["nx"] * case["images"]
        fft = 5 * case["nz"] * math.log2(case["nz"])
        return {"bytes": 4 * lines * (case["nz"] + m), "flops": lines * (2 * fft + 12 * m)}
    if case["path"] == "batch":
        parts = [work(f) for f in _batch_frames(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    ntx, nrx, np_ = _counts(case)
    f = case["frames"]
    esize = 4 if case["data"] == "float32" else 2
    live = _live_share(case) * nrx * np_           # (receive, pixel) pairs
    taps = live * ntx
    per = {"cubic": 20, "linear": 12, "nearest": 8}[case["interp"]]
    synthetic = case["path"] in ("synthetic", "slsc", "matrix", "grad_slow")
    out = {"tx_and_rx": np_, "tx_only": nrx * np_, "rx_only": ntx * np_}[case["sumtype"]]
    if case["path"] in ("dmas", "slsc"):
        out = np_
    rf = ntx * nrx * case["nt"]
    nbytes = f * (rf * esize + 4 * out)
    nbytes += 4 * np_ * (3 if case["path"] == "matrix" else 2) if synthetic else \
        8 * (ntx + nrx) * np_
    # what does not depend on the frame (delay, weight, knot: 8) and what does
    flops = taps * (8 + f * (per - 8)) if per > 8 else taps * (6 + 2 * f)
    flops += 13 * (ntx + nrx) * np_ if synthetic else 0
    if case["path"] == "dmas":
        flops += 4 * case["lags"] * live
    if case["path"] == "slsc":
        flops += live * (2 * case["nkern"] + 1) * (2 * case["nlag"] + 4)
    if case["path"] == "grad":
        nbytes += 4 * (out + rf + (ntx + nrx) * np_)
        flops += 26 * taps
    if case["path"] == "grad_slow":
        nbytes += 4 * (out + rf + 2 * np_)
        flops += 26 * taps
    return {"bytes": float(nbytes), "flops": float(flops)}


# ---------------------------------------------------------------------------
# the same in 64 bits, in plain torch
# ---------------------------------------------------------------------------
F64 = torch.float64


def _spline64(y):
    """(y, z) with a zero after the last sample: z_i = y''_i dt^2 / 6 of the natural cubic
    spline, 0.5 z_i-1 + 2 z_i + 0.5 z_i+1 = (y_i-1 - 2 y_i + y_i+1) / 2."""
    d = 0.5 * (y[..., 2:] - 2.0 * y[..., 1:-1] + y[..., :-2])
    z = torch.zeros_like(y)
    z[..., 1:-1] = _solve(d)
    pad = torch.zeros_like(y[..., :1])
    return torch.cat([y, pad], -1), torch.cat([z, pad], -1)


def _solve(d):
    """T^-1 d along the last axis, T = tridiagonal (0.5, 2, 0.5)."""
    n = d.shape[-1]
    v = d.movedim(-1, 0).contiguous()
    cp, m = [0.0] * n, [2.0] * n
    for i in range(n):
        m[i] = 2.0 - (0.5 * cp[i - 1] if i else 0.0)
        cp[i] = 0.5 / m[i]
        v[i].div_(m[i])
        if i:
            v[i].sub_(v[i - 1], alpha=0.5 / m[i])
    for i in range(n - 2, -1, -1):
        v[i].sub_(v[i + 1], alpha=cp[i])
    return v.movedim(0, -1)


def _points(geo, side, pnts, dtype):
    """Signed distances, projections and the acceptance test of every (point, pixel)."""
    t = lambda v: torch.as_tensor(v, device="cuda").to(torch.float32).to(dtype)  # noqa: E731
    o, n = t(geo["ovec" + side]), t(geo["nvec" + side])
    m2 = pr = None
    for k in range(pnts.shape[1]):
        d = pnts[:, k] - o[:, k, None]
        m2 = d * d if m2 is None else m2 + d * d
        pr = d * n[:, k, None] if pr is None else pr + d * n[:, k, None]
    return torch.sqrt(m2), pr


def _synthetic_delays(geo, dtype):
    """Transmit and receive delays and masks (no depth of field), in dtype arithmetic from
    the float32 arguments; alatx = 0 is a plane wave without a mask."""
    t = lambda v: torch.as_tensor(v, device="cuda").to(torch.float32).to(dtype)  # noqa: E731
    pnts, c0 = t(geo["pnts"]), float(np.float32(geo["c0"]))
    mag, pr = _points(geo, "tx", pnts, dtype)
    if float(np.max(np.abs(geo["alatx"]))) == 0.0:
        ttx, mtx = pr / c0, torch.ones_like(pr, dtype=torch.bool)
        dtx = pr
    else:
        dtx = torch.where(pr > 0, mag, -mag)
        ttx = dtx / c0 + t(geo["t0tx"])[:, None]
        mtx = (pr / mag).abs() >= t(np.cos(np.float32(geo["alatx"]).astype(np.float64)))[:, None]
    mag, pr = _points(geo, "rx", pnts, dtype)
    mrx = (pr / mag) >= t(np.cos(np.float32(geo["alarx"]).astype(np.float64)))[:, None]
    return ttx, mtx, mag / c0, mrx, dtx, mag


class _Taps:
    """The taps of one case: 32-bit decisions (range, weight, nearest sample), 64-bit values."""

    def __init__(self, case, slow=None):
        self.case = case
        self.dt32, self.dt = np.float32(1.0 / case["fs"]), float(np.float32(1.0 / case["fs"]))
        self.nt = case["nt"]
        self.xmax = float(np.float32(self.dt32 * np.float32(self.nt - 1)))
        if case["path"] in ("tabbed", "dmas", "grad"):
            self.ttx32, self.atx, self.trx32, self.arx = _tables(case)
            self.ttx, self.trx = self.ttx32.to(F64), self.trx32.to(F64)
            self.synthetic = False
        else:
            geo = _geometry(case)
            self.ttx32, self.mtx, self.trx32, self.mrx, d32, r32 = _synthetic_delays(
                geo, torch.float32)
            self.ttx, _, self.trx, _, self.dtx, self.drx = _synthetic_delays(geo, F64)
            if slow is not None:
                self.ttx32, self.trx32 = d32 * slow, r32 * slow
                self.ttx, self.trx = self.dtx * slow.to(F64), self.drx * slow.to(F64)
            self.synthetic = True
        self.ntx, self.nrx, self.np = self.ttx.shape[0], self.trx.shape[0], self.ttx.shape[1]

    def of(self, t, r):
        """(knot, fraction, weight) of transmit t and receives r (a slice), (nr, np) each;
        the weight is zero where the tap does not count."""
        x32 = self.ttx32[t] + self.trx32[r]
        ok = (x32 >= 0.0) & (x32 <= self.xmax)
        if self.synthetic:
            ok &= self.mtx[t] & self.mrx[r]
            w = ok.to(F64)
        else:
            ok &= (self.atx[t] * self.arx[r]).abs() >= THRESH
            w = torch.where(ok, self.atx[t].to(F64) * self.arx[r].to(F64), 0.0)
        if self.case["interp"] == "nearest":
            q32 = x32 / torch.tensor(self.dt32, device="cuda")
            j = (q32 + 0.5).to(torch.int64)
            inside = (j >= 0) & (j < self.nt)
            if not self.synthetic:
                w = torch.where(inside & ((self.atx[t] * self.arx[r]).abs() >= THRESH),
                                self.atx[t].to(F64) * self.arx[r].to(F64), 0.0)
            return j.clamp(0, self.nt - 1), None, w
        q = (self.ttx[t] + self.trx[r]) / self.dt
        j = torch.nan_to_num(torch.floor(q), 0.0, 0.0, 0.0).clamp(0, self.nt - 1)
        b = torch.nan_to_num(q - j, 0.0, 0.0, 0.0)
        return j.to(torch.int64), b, w

    def chunks(self):
        n = max(1, int(6e7 // self.np))
        for r0 in range(0, self.nrx, n):
            yield slice(r0, min(self.nrx, r0 + n))


def _value(case, b, y0, y1, z0, z1):
    if case["interp"] == "nearest":
        return y0
    if case["interp"] == "linear":
        return (1.0 - b) * y0 + b * y1
    a = 1.0 - b
    return a * y0 + b * y1 + (a * a * a - a) * z0 + (b * b * b - b) * z1


def _prefiltered(case, rf):
    """(y, z) of every channel, in 64 bits; z is zero where no spline is asked for."""
    if case["interp"] == "cubic":
        return _spline64(rf.to(F64))
    y = torch.nn.functional.pad(rf.to(F64), (0, 1))
    return y, torch.zeros_like(y)


def _das64(taps, rf, sumtype):
    """The image of every frame: rf (frames, ntx, nrx, nt)."""
    py, pz = _prefiltered(taps.case, rf)
    shape = {"tx_and_rx": (taps.np,), "tx_only": (taps.nrx, taps.np),
             "rx_only": (taps.ntx, taps.np)}[sumtype]
    out = torch.zeros((rf.shape[0],) + shape, dtype=F64, device="cuda")
    for r in taps.chunks():
        for t in range(taps.ntx):
            j, b, w = taps.of(t, r)
            j1 = j + 1
            for f in range(rf.shape[0]):
                y, z = py[f, t, r], pz[f, t, r]
                g = torch.gather
                v = w * _value(taps.case, b, g(y, 1, j), g(y, 1, j1), g(z, 1, j), g(z, 1, j1))
                if sumtype == "tx_and_rx":
                    out[f] += v.sum(0)
                elif sumtype == "tx_only":
                    out[f, r] += v
                else:
                    out[f, t] += v.sum(0)
    return out


def _gradients64(taps, rf, gout):
    """Image, dL/drf, and per (transmit, receive, pixel) dL/dx summed as the case asks."""
    case = taps.case
    py, pz = _prefiltered(case, rf)
    each = case["sumtype"] == "tx_only"
    img = torch.zeros((taps.nrx, taps.np) if each else (taps.np,), dtype=F64, device="cuda")
    gy, gz = torch.zeros_like(py), torch.zeros_like(pz)
    gtx = torch.zeros((taps.ntx, taps.np), dtype=F64, device="cuda")
    grx = torch.zeros((taps.nrx, taps.np), dtype=F64, device="cuda")
    gs = torch.zeros(taps.np, dtype=F64, device="cuda")
    g64 = gout.to(F64)
    for r in taps.chunks():
        up = g64[r] if each else g64[None]
        for t in range(taps.ntx):
            j, b, w = taps.of(t, r)
            j1, a = j + 1, 1.0 - b
            y, z = py[t, r], pz[t, r]
            y0, y1, z0, z1 = y.gather(1, j), y.gather(1, j1), z.gather(1, j), z.gather(1, j1)
            v = w * _value(case, b, y0, y1, z0, z1)
            if each:
                img[r] += v
            else:
                img += v.sum(0)
            slope = (y1 - y0 + (3 * b * b - 1) * z1 - (3 * a * a - 1) * z0) / taps.dt
            dx = w * up * slope
            gtx[t] += dx.sum(0)
            grx[r] += dx
            if taps.synthetic:
                gs += (dx * (taps.dtx[t] + taps.drx[r])).sum(0)
            wu = w * up
            gy[t, r] = gy[t, r].scatter_add(1, j, wu * a).scatter_add(1, j1, wu * b)
            gz[t, r] = gz[t, r].scatter_add(1, j, wu * (a ** 3 - a)).scatter_add(
                1, j1, wu * (b ** 3 - b))
    nt = taps.nt
    v = torch.zeros_like(gy[..., :nt])
    v[..., 1:-1] = _solve(gz[..., 1:nt - 1])
    lap = -2.0 * v
    lap[..., 1:] += v[..., :-1]
    lap[..., :-1] += v[..., 1:]
    return img, gy[..., :nt] + 0.5 * lap, gtx, grx, gs


def _slsc64(case, sep, mask):
    """Mean over lags of the mean normalised correlation of the kept elements' kernels.  The
    f-number mask keeps a run of consecutive elements, so lags count elements."""
    nx, nz, k, nlag = case["nx"], case["nz"], case["nkern"], case["nlag"]
    out = torch.empty((nx, nz), dtype=F64, device="cuda")
    sep, mask = sep.reshape(-1, nx, nz), mask.reshape(-1, nx, nz)
    iz = torch.arange(nz, device="cuda")[:, None] + torch.arange(-k, k + 1, device="cuda")
    inside = (iz >= 0) & (iz < nz)
    iz = iz.clamp(0, nz - 1)
    length = inside.sum(1).to(F64)
    for x in range(nx):
        v = torch.where(inside, sep[:, x][:, iz], 0.0)                     # (nrx, nz, 2k+1)
        kept = (mask[:, x][:, iz] | ~inside).all(-1)
        v = torch.where(inside, v - (v.sum(-1) / length)[..., None], 0.0)
        sd = torch.sqrt((v * v).sum(-1) / length)
        ok = kept & (sd >= 1e-10)
        v = torch.where(ok[..., None], v / sd[..., None], 0.0)
        res = torch.zeros(nz, dtype=F64, device="cuda")
        for m in range(1, nlag + 1):
            pair = ok[:-m] & ok[m:]
            dot = (v[:-m] * v[m:]).sum(-1) / length
            res += torch.where(pair, dot, 0.0).sum(0) / pair.sum(0) / nlag
        out[x] = torch.where(kept.sum(0) >= nlag + 1, res, 0.0)
    return out


def _bmode64(case, x):
    x = x.to(F64).cpu().numpy()
    n = case["nz"]
    f = np.fft.rfftfreq(n, 1 / case["ks"])
    lo, hi = int(np.argmin(np.abs(f - case["kmin"]))), int(np.argmin(np.abs(f - case["kmax"]))) + 1
    m, alpha = hi - lo, 0.25
    i = np.arange(m, dtype=np.float64)
    taper = np.ones(m)
    if m > 1:
        width = int(np.floor(alpha * (m - 1) / 2.0))
        edge = 0.5 * (1 + np.cos(np.pi * (-1 + 2.0 * i[:width + 1] / alpha / (m - 1))))
        taper[:width + 1], taper[m - width - 1:] = edge, edge[::-1]
    spec = np.fft.ifftshift(np.fft.rfft(x, axis=-1)[..., lo:hi] * taper, axes=-1)
    env = np.abs(np.fft.ifft(spec, axis=-1))
    ref = np.percentile(env, 99, axis=(-2, -1), keepdims=True)
    return torch.as_tensor(20 * np.log10(env / ref + 1e-10))


def exact(case, seed):
    gen = _seeded(seed)
    if case["path"] == "bmode":
        return _bmode64(case, _image_lines(case, gen))
    if case["path"] == "batch":
        frames = _batch_frames(case)
        rf = [_channels(_rf_shape(f), f["data"], gen) for f in frames]
        return [_das64(_Taps(f), v[None], "tx_and_rx")[0] for f, v in zip(frames, rf)]
    rf = _channels(_rf_shape(case), case["data"], gen)
    if case["path"] == "grad":
        gout = torch.randn(_grad_shape(case), generator=gen, device="cuda")
        img, grf, gtx, grx, _ = _gradients64(_Taps(case), rf, gout)
        return {"image": img, "rf": grf, "tautx": gtx, "taurx": grx}
    if case["path"] == "grad_slow":
        slow = _slowness(case, gen)
        gout = torch.randn(_grad_shape(case), generator=gen, device="cuda")
        img, grf, _, _, gs = _gradients64(_Taps(case, slow), rf, gout)
        return {"image": img, "rf": grf, "slowness": gs}
    taps = _Taps(case)
    rf4 = rf if rf.ndim == 4 else rf[None]
    if case["path"] == "slsc":
        return _slsc64(case, _das64(taps, rf4, "tx_only")[0], taps.mrx)
    if case["path"] == "dmas":
        sep = _das64(taps, rf4, "tx_only")[0]
        out = torch.zeros(taps.np, dtype=F64, device="cuda")
        for lag in range(1, case["lags"] + 1):
            p = sep[:-lag] * sep[lag:]
            out += (p if case["dmastype"] == "power" else p.sign() * p.abs().sqrt()).sum(0)
        return out
    out = _das64(taps, rf4, case["sumtype"])
    return out if rf.ndim == 4 else out[0]
