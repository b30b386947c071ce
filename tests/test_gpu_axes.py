"""Sums over transmits on the axes without 32-bit, unclamped knots (GPU): float32 delays in
steps of more than two samples, and 2^29 samples a transmit and more."""
import ctypes as ct

import numpy as np
import pytest
import torch

import pycbf_gb300 as pg
from gpu_util import assert_image_close
from oracle import oracle
from pycbf_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["cubic", "linear", "nearest"])
@pytest.mark.parametrize("sumtype", ["tx_and_rx", "tx_only"])
@pytest.mark.parametrize("ntx", [1, 5, 12, 13, 30, 453])
def test_coarse_axes_against_the_oracle(kind, sumtype, ntx):
    """From 1 s at 55 ns, 2.17 samples a step of the delays, some past both ends of the
    record; transmits in registers, in a padded and in an unpadded column.  (The knots next
    to such a delay round to it, so the cubic and linear images are zeros.)"""
    nrx, npx, nt, t0, dt = 7, 150, 492, 1.0, 5.5e-8
    r = np.random.default_rng(ntx)
    span = nt * dt
    f32 = lambda a: np.asarray(a, np.float32)
    tautx, taurx = f32(t0 + r.uniform(-0.1, 0.7, (ntx, npx)) * span), f32(r.uniform(0, 0.5, (nrx, npx)) * span)
    tautx[0, ::7] = np.nan
    apodtx, apodrx = f32(r.uniform(-1, 1, (ntx, npx))), f32(r.choice([0, 0.012, 1], (nrx, npx)))
    rf = f32(r.standard_normal((ntx, nrx, nt)))
    bf = pg.TabbedBeamformer(tautx=tautx, taurx=taurx, apodtx=apodtx, apodrx=apodrx, t0=t0, dt=dt, nt=nt,
                             interp={"kind": kind}, sumtype=sumtype, stage_channels=False)
    # a NaN delay never counts: to the oracle, one before the record
    ref = oracle.das_tabbed(rf, np.nan_to_num(tautx, nan=0.0), apodtx, taurx, apodrx, t0, dt, nt, interp=kind, sumtype=sumtype)
    assert (np.abs(ref).max() > 0) == (kind == "nearest")
    assert_image_close(bf(rf), ref)


def _per_receive(info, interp, rf, tables, npx):
    """Per-receive sums of rf by the C entry point (no beamformer: its float64 tables of
    30,000 receives are not needed)."""
    L = _lib.load()
    nws = L.pycbf_gb_workspace_bytes(ct.byref(info), interp)
    ws = torch.empty(nws, dtype=torch.uint8, device="cuda")
    out = torch.full((info.nrx, npx), float("nan"), device="cuda")
    _lib.check(L.pycbf_gb_das_tabbed(
        ct.byref(info), _lib.ptr(rf), *(_lib.ptr(t) for t in tables), npx, None, interp, 0.01,
        _lib.SUMTYPE["tx_only"], None, _lib.ptr(out), _lib.ptr(ws), nws, _lib.stream()), "das_tabbed")
    return out


@pytest.mark.parametrize("kind,ntx,nrx,nt", [("linear", 3, 129, 4194303), ("nearest", 3, 129, 4194303),
                                             ("linear", 13, 129, 4194303), ("cubic", 2, 29828, 18000)])
def test_long_records_give_the_rows_of_short_ones(kind, ntx, nrx, nt):
    """A transmit's channels are 2^29 samples or more: the per-receive sums of the last 9
    receives are those of a call with these receives alone, bit for bit."""
    assert nrx * nt >= 1 << 29
    npx, dt, few = 70, 4e-8, 9
    gen = torch.Generator(device="cuda").manual_seed(ntx)
    u = lambda n, a, b: torch.empty((n, npx), device="cuda").uniform_(a, b, generator=gen)
    tables = [u(ntx, -0.1 * nt * dt, 0.6 * nt * dt), u(ntx, 0.5, 1), u(nrx, 0, 0.5 * nt * dt), u(nrx, 0, 1)]
    rf = torch.empty((ntx, nrx, nt), device="cuda").normal_(generator=gen)
    info = lambda n: _lib.RFInfo(ntx, n, 0, 0.0, float(np.float32(dt)), nt, 1, _lib.F32)
    interp = _lib.INTERP[kind]
    rows = _per_receive(info(nrx), interp, rf, tables, npx)[-few:].clone()
    torch.cuda.empty_cache()
    part = [t[-few:].contiguous() if t.shape[0] == nrx else t for t in tables]
    want = _per_receive(info(few), interp, rf[:, -few:].contiguous(), part, npx)
    assert float(want.abs().max()) > 0 and torch.equal(rows, want)
    del rf, rows, want
    torch.cuda.empty_cache()


@pytest.mark.parametrize("kind", ["cubic", "linear", "nearest"])
@pytest.mark.parametrize("storage", ["float32", "float16"])
@pytest.mark.parametrize("staged", [True, False])
@pytest.mark.parametrize("wide", [0.02, 0.5])
def test_coarse_axes_gather_the_records_of_the_taps(kind, storage, staged, wide):
    """The images above cannot tell which records a cubic or linear sum read; NaN samples
    can: 0 x NaN shows in exactly the pixels and receives whose taps ('none', decided one
    by one) read a record of theirs.  With a staging plan (windows that fit a stage, and
    longer ones that do not) and without."""
    ntx, nrx, npx, nt, t0, dt = 5, 70, 333, 2072, 1.0, 5.5e-8
    r = np.random.default_rng(3)
    span = nt * dt
    kw = dict(tautx=t0 + r.uniform(-0.05, 0.6) * span + r.uniform(0, wide, (ntx, npx)) * span,
              taurx=r.uniform(0, 0.3, (nrx, 1)) * span + r.uniform(0, 0.01, (nrx, npx)) * span,
              apodtx=r.uniform(-1, 1, (ntx, npx)), apodrx=r.choice([0.0, 0.012, 1.0], (nrx, npx)), t0=t0,
              dt=dt, nt=nt, interp={"kind": kind}, storage=storage, pixel_order="natural")
    rf = r.standard_normal((ntx, nrx, nt)).astype(np.float32)
    for ch in r.integers(0, ntx * nrx, 60):
        at = r.integers(0, nt)
        rf.reshape(-1, nt)[ch, at:at + 100] = np.nan
    rf = torch.as_tensor(rf, device="cuda").to(getattr(torch, storage))
    taps = pg.TabbedBeamformer(sumtype="none", **kw)(rf).reshape(ntx, nrx, npx)
    bf = pg.TabbedBeamformer(sumtype="tx_only", stage_channels=staged, **kw)
    rows = bf(rf).reshape(nrx, npx)
    want = np.isnan(taps).any(0)
    assert 0 < want.sum() < want.size
    np.testing.assert_array_equal(np.isnan(rows), want)
    if staged:
        assert bf.kernel_status() == 0
