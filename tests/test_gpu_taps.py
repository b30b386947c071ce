"""Sums over transmits against the same call's single taps (GPU): the packed decisions of
the summing kernels, padded and unpadded transmit columns, and time axes whose float32
delays are coarser than a sample."""
import numpy as np
import pytest
import torch

import pycbf_gb300 as pg

pytestmark = pytest.mark.gpu


def _case(ntx, nrx, npx, nt, t0, dt, seed):
    """Delays on and next to knots and half-knots, before, inside and past the record."""
    r = np.random.default_rng(seed)
    k = r.integers(-3, nt + 3, (ntx, npx)) + r.choice([0.0, 0.5, 0.25], (ntx, npx))
    x = (np.float32(t0) + np.float32(dt) * k.astype(np.float32)).astype(np.float32)
    x = np.where(r.uniform(size=x.shape) < 0.5, np.nextafter(x, np.float32(r.choice([-9e9, 9e9]))), x)
    return dict(tautx=x, taurx=np.zeros((nrx, npx)), apodtx=r.choice([0.0, 0.009, 0.01, -1.0], (ntx, npx)),
                apodrx=r.choice([0.0, 1.0, 1.1], (nrx, npx)), t0=t0, dt=dt, nt=nt)


@pytest.mark.parametrize("kind", ["cubic", "linear", "nearest"])
@pytest.mark.parametrize("storage", ["float32", "float16"])
@pytest.mark.parametrize("ntx,t0,dt", [(3, 1.3e-6, 4e-8), (13, 0.0, 1e-7), (453, 2e-7, 4e-8),
                                       (454, 0.0, 4e-8), (7, 1.0, 2.561e-8), (14, 1.0, 1.1e-7)])
def test_sums_equal_their_single_taps(kind, storage, ntx, t0, dt):
    """float32 sums of at most 454 x 2 taps: 1e-5 of the sum of magnitudes (16-bit
    records round the same way in both)."""
    case = _case(ntx, 2, 133, 64, t0, dt, ntx)
    kw = dict(interp={"kind": kind}, storage=storage, stage_channels=False)
    dtype = {"float32": torch.float32, "float16": torch.float16}[storage]
    g = torch.Generator(device="cuda").manual_seed(1)
    rf = torch.randn((ntx, 2, 64), generator=g, device="cuda").to(dtype)
    taps = pg.TabbedBeamformer(sumtype="none", **case, **kw)(rf, out_as_numpy=False).double()
    got = pg.TabbedBeamformer(**case, **kw)(rf, out_as_numpy=False).double()
    each = pg.TabbedBeamformer(sumtype="tx_only", **case, **kw)(rf, out_as_numpy=False).double()
    mag = taps.abs().sum((0, 1))
    # at 2.561e-8 s from 1 s every knot falls on its neighbours: cubic and linear weights are 0
    assert float(mag.max()) > 0 or (dt == 2.561e-8 and kind != "nearest")
    assert bool(((got - taps.sum((0, 1))).abs() <= 1e-5 * mag + 1e-30).all())
    assert bool(((each - taps.sum(0)).abs() <= 1e-5 * taps.abs().sum(0) + 1e-30).all())


@pytest.mark.parametrize("kind", ["cubic", "linear"])
@pytest.mark.parametrize("ntx", [3, 13, 40])
def test_nan_weights_drop_their_taps(kind, ntx):
    """A NaN weight among equal ones drops its tap, as a weight below the threshold does."""
    case = _case(ntx, 70, 133, 64, 1.3e-6, 4e-8, ntx)
    r = np.random.default_rng(ntx)
    bad = r.uniform(size=(ntx, 133)) < 0.2
    rf = r.standard_normal((3, ntx, 70, 64)).astype(np.float32)
    images = []
    for value in (np.nan, 0.0):
        case["apodtx"] = np.where(bad, value, 1.0)
        bf = pg.TabbedBeamformer(interp={"kind": kind}, stage_channels=False, **case)
        images.append([bf(rf), np.stack([bf(f) for f in rf])])
    assert np.abs(images[1][0]).max() > 0
    for a, b in zip(*images):
        np.testing.assert_array_equal(a, b)
