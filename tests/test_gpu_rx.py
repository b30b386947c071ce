"""Sums over transmits with the receives spread over the warps of a CTA (GPU): the order of
the sums, runs of receives and their remainders, ragged pixels, and the kernels that serve
the time axes without packed decisions."""
import numpy as np
import pytest
import torch

import pycbf_gb300 as pg
from pycbf_gb300 import adjoint

pytestmark = pytest.mark.gpu
DT = {"float32": torch.float32, "float16": torch.float16, "bfloat16": torch.bfloat16}


def _class(das, dmas, nrx, kw):
    if kw.get("sumtype") != "dmas":
        return das
    kw.update(sumtype="tx_only", lags=np.arange(1, nrx), lagaxis="rx", sumlags=True)
    return dmas


def _tabbed(ntx, nrx, npx, nt, seed, t0=1.3e-7, dt=4e-8, **kw):
    r = np.random.default_rng(seed)
    span = nt * dt
    return _class(pg.TabbedBeamformer, pg.TabbedDMASBeamformer, nrx, kw)(
        tautx=t0 + r.uniform(-0.1, 0.6, (ntx, npx)) * span, taurx=r.uniform(0, 0.6, (nrx, npx)) * span,
        apodtx=np.ones((ntx, npx)) if seed % 2 else r.uniform(-1, 1, (ntx, npx)),
        apodrx=r.choice([0.0, 0.01, 0.5, 1.0], (nrx, 1)) * r.uniform(0.5, 1, (nrx, npx)), t0=t0, dt=dt,
        nt=nt, **kw)


def _synthetic(ntx, nrx, npx, nt, seed, **kw):
    r = np.random.default_rng(seed)
    xe = 3e-4 * (np.arange(nrx) - (nrx - 1) / 2)
    src = np.stack([r.uniform(-4e-3, 4e-3, ntx), np.full(ntx, -8e-3)], 1)
    up = np.array([0.0, 1.0])
    pnts = np.stack([r.uniform(xe[0], xe[-1] + 1e-4, npx), r.uniform(1e-3, 25e-3, npx)], 1)
    return _class(pg.SyntheticBeamformer, pg.SyntheticDMASBeamformer, nrx, kw)(
        ovectx=src, nvectx=np.tile(up, (ntx, 1)), doftx=np.zeros(ntx), alatx=np.full(ntx, 0.9),
        t0tx=np.full(ntx, -8e-3 / 1540), ovecrx=np.stack([xe, np.zeros(nrx)], 1),
        nvecrx=np.tile(up, (nrx, 1)), alarx=np.full(nrx, 0.45), c0=1540.0, pnts=pnts, t0=0.0, dt=4e-8,
        nt=nt, **kw)


def _channels(bf, seed, n=0, dtype=torch.float32):
    g = torch.Generator(device="cuda").manual_seed(seed)
    shape = ((n,) if n else ()) + (bf.ntx, bf.nrx, bf.nt)
    return torch.randn(shape, generator=g, device="cuda").to(dtype)


def _block_sums(rows):
    """Image of each receive's sum, float32: blocks of 64 receives in order, then the blocks."""
    image = np.zeros(rows.shape[1:], np.float32)
    for r0 in range(0, rows.shape[0], 64):
        block = np.zeros_like(image)
        for row in rows[r0:r0 + 64]:
            block = block + row
        image = image + block
    return image


@pytest.mark.parametrize("make", [_tabbed, _synthetic])
@pytest.mark.parametrize("kind", ["cubic", "linear", "nearest"])
@pytest.mark.parametrize("ntx,nrx,npx", [(1, 1, 1), (3, 7, 31), (4, 64, 33), (13, 65, 257),
                                         (5, 257, 100), (30, 300, 64), (454, 9, 40)])
def test_images_add_the_receives_in_blocks(make, kind, ntx, nrx, npx):
    """Bit for bit; the image of DMAS (products of the receives' roots) in float64 to
    1e-5 of its terms' magnitudes (300 float32 fused multiply-adds)."""
    kw = dict(interp={"kind": kind})
    args = (ntx, nrx, npx, 301, ntx + nrx)
    rf = _channels(make(*args), 1)
    rows = make(*args, sumtype="tx_only", **kw)(rf).reshape(nrx, npx)
    np.testing.assert_array_equal(make(*args, **kw)(rf).reshape(npx), _block_sums(rows))
    s = np.sign(rows) * np.sqrt(np.abs(rows))
    if nrx == 1:
        return
    got = make(*args, sumtype="dmas", **kw)(rf).reshape(npx)
    want = ((s.sum(0, dtype=np.float64) ** 2) - (s.astype(np.float64) ** 2).sum(0)) / 2
    assert np.all(np.abs(got - want) <= 1e-5 * np.abs(s).sum(0, dtype=np.float64) ** 2 + 1e-12)


@pytest.mark.parametrize("make", [_tabbed, _synthetic])
@pytest.mark.parametrize("storage", ["float32", "float16", "bfloat16"])
@pytest.mark.parametrize("ntx,nrx,npx", [(2, 65, 33), (13, 129, 100), (40, 257, 31)])
def test_groups_of_frames_add_the_same_way(make, storage, ntx, nrx, npx):
    kw = dict(storage=storage)
    args = (ntx, nrx, npx, 301, ntx + nrx + 1)
    rf = _channels(make(*args, **kw), 2, 9, DT[storage])
    rows = make(*args, sumtype="tx_only", **kw)(rf).reshape(9, nrx, npx)
    images = make(*args, **kw)(rf).reshape(9, npx)
    one = make(*args, **kw)(rf[3]).reshape(npx)
    for f in range(9):
        np.testing.assert_array_equal(images[f], _block_sums(rows[f]))
    np.testing.assert_array_equal(images[3], one)


@pytest.mark.parametrize("kind", ["cubic", "linear", "nearest"])
@pytest.mark.parametrize("sumtype", ["tx_and_rx", "tx_only", "dmas"])
def test_coarse_axes_agree_with_and_without_a_plan(kind, sumtype):
    """Float32 delays from 1 s in steps below theirs: every tap decided exactly, by the
    staged kernel and by das_kernel alike."""
    args, kw = (5, 70, 333, 492, 4), dict(t0=1.0, dt=5.5e-8, interp={"kind": kind}, sumtype=sumtype)
    staged, plain = _tabbed(*args, **kw), _tabbed(*args, stage_channels=False, **kw)
    assert staged._plan is not None and plain._plan is None
    rf = _channels(plain, 3, 3)
    images = plain(rf)
    # the knots on either side of a delay round to it: cubic and linear weights are 0
    assert np.abs(images).max() > 0 or kind != "nearest"
    np.testing.assert_array_equal(staged(rf), images)
    np.testing.assert_array_equal(staged(rf[1]), images[1])
    assert staged.kernel_status() == 0


@pytest.mark.parametrize("ntx,nrx,npx", [(1, 1, 1), (3, 7, 31), (13, 65, 257), (30, 130, 33), (128, 9, 40)])
@pytest.mark.parametrize("sumtype", ["tx_and_rx", "tx_only"])
@pytest.mark.parametrize("dtype", ["float32", "float16"])
def test_delay_gradients_of_one_frame_and_of_several(ntx, nrx, npx, sumtype, dtype):
    """One frame's gradients, with the upstream gradient in the weights, against the same
    frame next to one whose gradient is zero, where the products are summed per tap: at
    most 1170 products in float32, 1170 x 2^-24 x 1.2 < 1e-4 of the largest; the slowness
    form likewise, and its image against its receives' sums bit for bit."""
    bf = _tabbed(ntx, nrx, npx, 301, ntx + nrx, pixel_order="natural")
    rf = _channels(bf, 4, 2, DT[dtype])
    apod = bf._tables[1], bf._tables[3]
    syn = _synthetic(ntx, nrx, npx, 301, ntx + nrx)
    slow0 = torch.full((npx,), 1 / 1500.0, device="cuda")
    kw = dict(t0=bf.t0, dt=bf.dt, thresh=bf.thresh, sumtype=sumtype)

    def grads(frames, make, *tables):
        leaves = [t.clone().requires_grad_(True) for t in tables]
        out = make(frames, *leaves)
        g = torch.randn(out.shape, generator=torch.Generator().manual_seed(5)).cuda()
        if frames.ndim == 4:
            g = torch.stack([torch.randn(out.shape[1:], generator=torch.Generator().manual_seed(5)).cuda(),
                             torch.zeros_like(out[1])])
        return torch.autograd.grad(out, leaves, g)

    tables = lambda f, ttx, trx: adjoint.das_tabbed(f, ttx, trx, *apod, **kw)
    slowness = lambda f, s: adjoint.das_synthetic_slowness(f, s, syn, sumtype=sumtype)
    for make, leaves in ((tables, (bf._tables[0], bf._tables[2])), (slowness, (slow0,))):
        for one, two in zip(grads(rf[0], make, *leaves), grads(rf, make, *leaves)):
            assert bool(((one - two).abs() <= 1e-4 * two.abs().max()).all())
    rows = adjoint.das_synthetic_slowness(rf[0], slow0, syn, sumtype="tx_only").cpu().numpy()
    image = adjoint.das_synthetic_slowness(rf[0], slow0, syn, sumtype="tx_and_rx").cpu().numpy()
    np.testing.assert_array_equal(image, _block_sums(rows.reshape(nrx, npx)))


@pytest.mark.parametrize("ntx,nrx,npx,nt", [(2, 1, 5000, 16), (1, 1, 1, 2), (3, 7, 300, 301), (5, 33, 4000, 64)])
@pytest.mark.parametrize("sumtype", ["tx_and_rx", "tx_only"])
@pytest.mark.parametrize("make", [_tabbed, _synthetic])
def test_channel_gradients_in_the_least_workspace(ntx, nrx, npx, nt, sumtype, make, monkeypatch):
    """With and without room for the delay ranges and tables: the same sums over other
    parts, at most 5000 taps a sample in float32 (1e-5 of the largest sum)."""
    bf = make(ntx, nrx, npx, nt, ntx + nrx)
    rf = _channels(bf, 6)
    slow = torch.full((npx,), 1 / 1540.0, device="cuda")

    def grad():
        x = rf.clone().requires_grad_(True)
        out = (adjoint.das_synthetic_slowness(x, slow, bf, sumtype=sumtype) if make is _synthetic
               else bf.differentiable(x, sumtype=sumtype))
        g = torch.randn(out.shape, generator=torch.Generator().manual_seed(7)).cuda()
        return torch.autograd.grad(out, x, g)[0]

    full = grad()
    def least(L, info, np_, synthetic, device):
        n = L.pycbf_gb_adjoint_workspace_bytes(info, np_)
        return torch.empty(n, dtype=torch.uint8, device=device), n
    monkeypatch.setattr(adjoint, "_workspace", least)
    assert bool(((grad() - full).abs() <= 1e-5 * full.abs().max()).all())
