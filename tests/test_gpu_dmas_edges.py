"""Delay-multiply-and-sum at the edges of its kernels (GPU)."""
import numpy as np
import pytest
import torch

import pycbf_gb300 as pg
from pycbf_gb300 import _lib

pytestmark = pytest.mark.gpu
BIG = 3e38


def _fused(geometry, kind, npx=64, nrx=4, **kw):
    """All lags summed: receive 2 reaches the odd pixels only, every receive in range."""
    nt = 64
    common = dict(nt=nt, interp={"kind": kind}, lags=np.arange(1, nrx), lagaxis="rx", sumlags=True, **kw)
    if geometry == "tabbed":
        t0, dt = common.pop("axis", (0.0, 4e-8))
        apodrx = np.ones((nrx, npx))
        apodrx[2, ::2] = 0
        return pg.TabbedDMASBeamformer(
            tautx=np.full((2, npx), t0 + 10.5 * dt), taurx=np.full((nrx, npx), 20 * dt),
            apodtx=np.ones((2, npx)), apodrx=apodrx, t0=t0, dt=dt, **common)
    x = np.where(np.arange(npx) % 2, 0.0, 2e-3)
    alarx = np.full(nrx, 1.5)
    alarx[2] = 0.1
    up, zero = np.array([0.0, 1.0]), np.zeros((2, 2))
    return pg.SyntheticDMASBeamformer(
        ovectx=zero, nvectx=np.tile(up, (2, 1)), doftx=np.zeros(2), alatx=np.zeros(2), t0tx=np.zeros(2),
        ovecrx=np.zeros((nrx, 2)), nvecrx=np.tile(up, (nrx, 1)), alarx=alarx, c0=1540.0,
        pnts=np.stack([x, np.full(npx, 3e-3)], 1), t0=0.0, dt=2e-7, **common)


@pytest.mark.parametrize("dmastype", ["ssr", "power"])
@pytest.mark.parametrize("geometry,kind,kw", [
    ("tabbed", "cubic", {}), ("tabbed", "linear", {}), ("tabbed", "nearest", {}),
    ("tabbed", "cubic", dict(nframes=2)), ("tabbed", "nearest", dict(axis=(1.0, 5.5e-8))),
    ("tabbed", "nearest", dict(axis=(1.0, 5.5e-8), stage_channels=False)),
    ("synthetic", "cubic", {}), ("synthetic", "linear", {}), ("synthetic", "cubic", dict(nframes=2))])
def test_masked_receive_after_an_infinite_sum(geometry, kind, kw, dmastype):
    """Receive 1's sum over two transmits overflows.  Its products with the positive sums
    around it are infinite; receive 2, where masked, takes no part (0 x inf would be NaN)."""
    kw = dict(kw)
    nframes = kw.pop("nframes", 0)
    bf = _fused(geometry, kind, dmastype=dmastype, **kw)
    assert bf._fused
    rf = torch.ones(((nframes,) if nframes else ()) + (bf.ntx, bf.nrx, bf.nt), device="cuda")
    rf[..., 1, :] = BIG
    out = bf(rf, out_as_numpy=False)
    assert bool((out == float("inf")).all())


@pytest.mark.parametrize("lags", [[40], [30, 60], [0, 1, 25], [-1, 24, 200, 5], [24, 24, 1],
                                  list(range(10, 26)), list(range(60))])
@pytest.mark.parametrize("nsep", [1, 7, 8, 41, 128])
@pytest.mark.parametrize("power", [0, 1])
@pytest.mark.parametrize("sumlags", [0, 1])
def test_lag_lists_of_any_length(lags, nsep, power, sumlags):
    """Lists within and beyond the short kernel's lags, with lags that have no pairs, two
    frames: at most nsep float32 additions a lag and 60 lags, each product and root rounded
    a few times, (nsep + 70) 2^-24 of the magnitudes."""
    npx, nf = 131, 2
    gen = torch.Generator(device="cuda").manual_seed(nsep)
    im = torch.randn((nf, nsep, npx), generator=gen, device="cuda")
    out = torch.full((nf, npx) if sumlags else (nf, len(lags), npx), float("nan"), device="cuda")
    dev = torch.as_tensor(lags, dtype=torch.int32, device="cuda")
    L = _lib.load()
    _lib.check(L.pycbf_gb_dmas(_lib.ptr(im), nf, nsep, npx, _lib.ptr(dev), len(lags), power, sumlags,
                               _lib.ptr(out), _lib.stream()), "dmas")
    x = im.double()
    want, size = [], []
    for lag in lags:
        n = max(nsep - lag, 0) if lag >= 0 else 0
        p = x[:, :n] * x[:, nsep - n:]
        t = p if power else p.sign() * p.abs().sqrt()
        want.append(t.sum(1))
        size.append(t.abs().sum(1))
    want, size = torch.stack(want, 1), torch.stack(size, 1)
    if sumlags:
        want, size = want.sum(1), size.sum(1)
    assert bool(((out.double() - want).abs() <= (nsep + 70) * 2.0 ** -24 * size).all())
