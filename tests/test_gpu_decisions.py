"""Sums over transmits against the sums of their taps (GPU): das_rx_kernel and the kernel of
several frames decide taps two at a time; sumtype 'none' writes every tap, decided one by
one by other code."""
import numpy as np
import pytest
import torch

import pycbf_gb300 as pg
from test_gpu_rx import DT

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,storage,frames", [
    ("cubic", "float32", 1), ("cubic", "float16", 1), ("cubic", "bfloat16", 1), ("linear", "float32", 1),
    ("linear", "float16", 1), ("linear", "bfloat16", 1), ("nearest", "float32", 1), ("nearest", "float16", 1),
    ("cubic", "float32", 2), ("cubic", "float32", 4), ("cubic", "float16", 8), ("cubic", "bfloat16", 3)])
@pytest.mark.parametrize("ntx,nrx,npx", [(1, 1, 33), (4, 65, 70), (11, 130, 257), (30, 9, 100)])
def test_sums_are_those_of_their_taps(kind, storage, frames, ntx, nrx, npx):
    """Delays on and next to the samples and half-samples, before, at and past both ends,
    NaN and infinite; weights on either side of the threshold, NaN among them.  A tap's value
    is at most |w| times 4 samples' worth of products, each rounded a few times, and
    ntx of them are added in float32: (ntx + 8) 2^-22 of them all."""
    nt, t0, dt, thresh = 301, 1.3e-7, 4e-8, 0.01
    r = np.random.default_rng(ntx + nrx)
    f32 = lambda a: np.asarray(a, np.float32)
    quant = lambda lo, hi, shape: (r.integers(2 * lo, 2 * hi, shape) / 2 + r.choice([0, 0, 1e-4, -1e-4, 0.3], shape))
    tautx, taurx = f32(t0 + dt * quant(-30, 200, (ntx, npx))), f32(dt * quant(0, 140, (nrx, npx)))
    for table in (tautx, taurx):
        table[r.random(table.shape) < 0.02] = np.nan
        table[r.random(table.shape) < 0.02] = np.inf
    apodtx = f32(r.choice([1.0, 0.1, -0.1, 0.0], (ntx, npx)))
    apodtx[r.random(apodtx.shape) < 0.02] = np.nan
    edge = np.nextafter(np.float32(0.1), np.float32(1))
    apodrx = f32(r.choice([1.0, 0.1, float(edge), 0.0999, 0.01, -0.5, 0.0], (nrx, npx)))
    kw = dict(tautx=tautx, taurx=taurx, apodtx=apodtx, apodrx=apodrx, t0=t0, dt=dt, nt=nt, thresh=thresh,
              interp={"kind": kind}, storage=storage)
    rf = torch.as_tensor(r.standard_normal((frames, ntx, nrx, nt)), dtype=torch.float32).to(DT[storage]).cuda()
    taps = pg.TabbedBeamformer(sumtype="none", **kw)(rf).reshape(frames, ntx, nrx, npx).astype(np.float64)
    assert np.abs(taps).max() > 0
    weight = (np.abs(apodtx)[:, None] * np.abs(apodrx)[None]).astype(np.float64)
    bound = (ntx + 8) * 2.0 ** -22 * 4 * float(rf.float().abs().max()) * np.nansum(weight, 0)
    rows = pg.TabbedBeamformer(sumtype="tx_only", **kw)(rf).reshape(frames, nrx, npx)
    assert np.all(np.abs(rows - taps.sum(1)) <= bound)
    image = pg.TabbedBeamformer(sumtype="tx_and_rx", **kw)(rf).reshape(frames, npx)
    total = (nrx + 8) * 2.0 ** -23 * np.abs(taps).sum((1, 2)) + bound.sum(0)
    assert np.all(np.abs(image - taps.sum((1, 2))) <= total)


@pytest.mark.parametrize("kind,storage,frames", [
    ("cubic", "float32", 1), ("cubic", "float16", 1), ("linear", "float32", 1), ("linear", "bfloat16", 1),
    ("nearest", "float32", 1), ("cubic", "float32", 3), ("cubic", "float16", 2)])
@pytest.mark.parametrize("sumtype", ["tx_only", "tx_and_rx"])
@pytest.mark.parametrize("ones", [False, True])
@pytest.mark.parametrize("ntx,nrx,npx", [(1, 1, 129), (12, 2, 40), (13, 1, 300), (75, 2, 131), (302, 1, 65), (454, 2, 33)])
def test_few_receives_give_the_rows_of_more(kind, storage, frames, sumtype, ones, ntx, nrx, npx):
    """One and two receives go to another kernel than three: the sums of a call whose
    further receives have no weight, bit for bit."""
    nt, dt = 301, 4e-8
    r = np.random.default_rng(ntx)
    more = 3
    taurx, apodrx = r.uniform(0, 140, (more, npx)) * dt, r.choice([0.0, 0.012, 1.0], (more, npx))
    apodrx[nrx:] = 0
    tautx = r.uniform(-30, 200, (ntx, npx)) * dt
    apodtx = np.ones((ntx, npx)) if ones else r.uniform(-1, 1, (ntx, npx))
    rf = torch.as_tensor(r.standard_normal((frames, ntx, more, nt)), dtype=torch.float32).to(DT[storage]).cuda()
    kw = dict(tautx=tautx, apodtx=apodtx, t0=0.0, dt=dt, nt=nt, interp={"kind": kind}, storage=storage,
              sumtype=sumtype)
    want = pg.TabbedBeamformer(taurx=taurx, apodrx=apodrx, **kw)(rf)
    got = pg.TabbedBeamformer(taurx=taurx[:nrx], apodrx=apodrx[:nrx], **kw)(rf[:, :, :nrx].contiguous())
    if sumtype == "tx_only":
        want = want.reshape(frames, more, npx)[:, :nrx]
    assert np.abs(got).max() > 0
    np.testing.assert_array_equal(got.reshape(want.shape), want)


@pytest.mark.parametrize("kind,storage,frames", [
    ("cubic", "float32", 1), ("cubic", "float16", 1), ("linear", "float32", 1), ("nearest", "float32", 1),
    ("nearest", "float32", 2), ("cubic", "float32", 2), ("cubic", "float16", 8)])
@pytest.mark.parametrize("geom,ntx,npx,few", [
    ("tabbed", 12, 16384, 2), ("tabbed", 13, 24575, 1), ("tabbed", 13, 24577, 2), ("tabbed", 140, 42624, 3),
    ("synthetic", 5, 40001, 4), ("synthetic", 31, 84630, 2)])
def test_receives_that_fit_one_thread_give_the_rows_of_more(kind, storage, frames, geom, ntx, npx, few):
    """How many receives one thread a pixel walks goes by the pixels and transmits; beyond, they
    are spread over warps: the sums per receive on both sides of that number, and the images
    as the sums of those, bit for bit."""
    nt, dt = 301, 4e-8
    r = np.random.default_rng(ntx)
    common = dict(t0=0.0, dt=dt, nt=nt, interp={"kind": kind}, storage=storage, pixel_order="natural")
    xe = 3e-4 * (np.arange(few + 1) - few / 2)
    tables = dict(tautx=r.uniform(-30, 200, (ntx, npx)) * dt, apodtx=r.uniform(-1, 1, (ntx, npx)))
    taurx, apodrx = r.uniform(0, 140, (few + 1, npx)) * dt, r.choice([0.0, 0.012, 1.0], (few + 1, npx))
    pnts = np.stack([r.uniform(-1e-3, 1e-3, npx), r.uniform(1e-3, 8e-3, npx)], 1)
    up = np.array([0.0, 1.0])

    def run(nrx, sumtype):
        if geom == "tabbed":
            bf = pg.TabbedBeamformer(taurx=taurx[:nrx], apodrx=apodrx[:nrx], sumtype=sumtype, **tables, **common)
        else:
            src = np.stack([np.linspace(-4e-3, 4e-3, ntx), np.full(ntx, -8e-3)], 1)
            bf = pg.SyntheticBeamformer(
                ovectx=src, nvectx=np.tile(up, (ntx, 1)), doftx=np.zeros(ntx), alatx=np.full(ntx, 0.9),
                t0tx=np.full(ntx, -8e-3 / 1540), ovecrx=np.stack([xe[:nrx], np.zeros(nrx)], 1),
                nvecrx=np.tile(up, (nrx, 1)), alarx=np.full(nrx, 0.45), c0=1540.0, pnts=pnts, sumtype=sumtype,
                **common)
        return bf(rf[:, :, :nrx].contiguous()).reshape((frames, nrx, npx) if sumtype == "tx_only" else (frames, npx))

    rf = torch.as_tensor(r.standard_normal((frames, ntx, few + 1, nt)), dtype=torch.float32).to(DT[storage]).cuda()
    more = run(few + 1, "tx_only")
    assert np.abs(more).max(axis=(0, 2)).min() > 0
    np.testing.assert_array_equal(run(few, "tx_only"), more[:, :few])
    for nrx in (few, few + 1):
        image = np.zeros((frames, npx), np.float32)
        for k in range(nrx):
            image = image + more[:, k]
        np.testing.assert_array_equal(run(nrx, "tx_and_rx"), image)
