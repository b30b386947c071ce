"""Several frames in one call: groups of frames share the decisions of a tap, and
every image equals the single-frame call's bit for bit (GPU)."""
import numpy as np
import pytest
import torch

import pycbf_gb300 as pg

pytestmark = pytest.mark.gpu
DT = {"float32": torch.float32, "float16": torch.float16, "bfloat16": torch.bfloat16}


def _tabbed(ntx, nrx, npx, nt, seed, **kw):
    """Delays around the record, some past either end, weights around the threshold."""
    r = np.random.default_rng(seed)
    dt = 4e-8
    span = nt * dt
    tx = np.sort(r.uniform(-0.05, 0.5, npx))[None] * span + r.uniform(0, 0.05, (ntx, 1)) * span
    rx = r.uniform(0, 0.6, (nrx, 1)) * span + np.linspace(0, 0.05, npx)[None] * span
    ones = kw.pop("ones", False)
    return pg.TabbedBeamformer(
        tautx=tx, taurx=rx, apodtx=np.ones((ntx, npx)) if ones else r.uniform(-1, 1, (ntx, npx)),
        apodrx=r.choice([0.0, 0.01, 0.02, 0.5, 1.0], (nrx, npx)), t0=1.3e-7, dt=dt, nt=nt, **kw)


def _synthetic(ntx, nrx, npx, nt, seed, cls=pg.SyntheticBeamformer, **kw):
    r = np.random.default_rng(seed)
    xe = 3e-4 * (np.arange(nrx) - (nrx - 1) / 2)
    src = np.stack([r.uniform(-4e-3, 4e-3, ntx), np.full(ntx, -8e-3)], 1)
    up = np.array([0.0, 1.0])
    pnts = np.stack([r.uniform(-6e-3, 6e-3, npx), r.uniform(1e-3, 25e-3, npx)], 1)
    return cls(ovectx=src, nvectx=np.tile(up, (ntx, 1)), doftx=np.zeros(ntx),
               alatx=np.full(ntx, 0.6), t0tx=np.full(ntx, -8e-3 / 1540),
               ovecrx=np.stack([xe, np.zeros(nrx)], 1), nvecrx=np.tile(up, (nrx, 1)),
               alarx=np.full(nrx, 0.45), c0=1540.0, pnts=pnts, t0=0.0, dt=4e-8, nt=nt, **kw)


def _frames(bf, n, seed, dtype=torch.float32):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn((n, bf.ntx, bf.nrx, bf.nt), generator=g, device="cuda").to(dtype)


def _same(bf, rf):
    many = bf(rf, out_as_numpy=False)
    for k in range(rf.shape[0]):
        one = bf(rf[k], out_as_numpy=False)
        assert float(one.abs().max()) > 0
        assert torch.equal(many[k], one), (k, float((many[k] - one).abs().max()))


@pytest.mark.parametrize("storage", ["float32", "float16", "bfloat16"])
@pytest.mark.parametrize("n", [2, 3, 5, 8, 13])
@pytest.mark.parametrize("make,ntx", [(_tabbed, 3), (_tabbed, 13), (_synthetic, 1), (_synthetic, 30)])
def test_frames_equal_single_frames(make, ntx, n, storage):
    bf = make(ntx, 67, 333, 513, ntx, storage=storage)
    _same(bf, _frames(bf, n, n, DT[storage]))


@pytest.mark.parametrize("kw", [dict(sumtype="tx_only"), dict(sumtype="rx_only"),
                                dict(sumtype="none"), dict(stage_channels=False),
                                dict(ones=True, stage_channels=False)])
def test_frames_sums_and_routes(kw):
    bf = _tabbed(5, 20, 200, 512, 3, **kw)
    for n in (4, 9):
        _same(bf, _frames(bf, n, n))


def test_frames_int16_and_dmas():
    bf = _tabbed(4, 33, 150, 600, 5, stage_channels=False)
    rf = (_frames(bf, 6, 1) * 1000).round().to(torch.int16)
    _same(bf, rf)
    for power in ("ssr", "power"):
        dm = _synthetic(7, 12, 140, 400, 6, cls=pg.SyntheticDMASBeamformer,
                        lags=np.arange(1, 12), dmastype=power)
        assert dm._fused
        _same(dm, _frames(dm, 5, 2))


@pytest.mark.parametrize("sumtype", ["tx_and_rx", "tx_only"])
def test_more_than_a_gigabyte_of_records_goes_by_receive_blocks(sumtype):
    bf = _synthetic(40, 200, 140, 2100, 7, sumtype=sumtype)
    _same(bf, _frames(bf, 4, 3))


@pytest.mark.parametrize("lags", [[1], [0, 2, 5], list(range(1, 9)), [31, 1, -3, 7, 30],
                                  list(range(1, 17)), [1, 32], list(range(1, 18)), [40]])
@pytest.mark.parametrize("nsep,npx", [(1, 5), (7, 300), (33, 128), (70, 131)])
@pytest.mark.parametrize("power,sumlags", [(0, 1), (1, 1), (0, 0)])
def test_dmas_lag_lists(lags, nsep, npx, power, sumlags):
    """Short lags (one walk with a ring) and any others, against float64 sums: at most
    70 products of at most 16 lags, each rounded a few times: 100 ulp of the sum of
    their magnitudes."""
    import ctypes as ct

    from pycbf_gb300 import _lib
    im = torch.randn((2, nsep, npx), device="cuda")
    lg = torch.tensor(lags, dtype=torch.int32, device="cuda")
    out = torch.empty((2, npx) if sumlags else (2, len(lags), npx), device="cuda")
    p = lambda t: ct.c_void_p(t.data_ptr())  # noqa: E731
    L = _lib.load()
    _lib.check(L.pycbf_gb_dmas(p(im), 2, nsep, npx, p(lg), len(lags), power, sumlags, p(out),
                               ct.c_void_p(torch.cuda.current_stream().cuda_stream)), "dmas")
    x = im.double()
    ref = torch.zeros((2, len(lags), npx), dtype=torch.float64, device="cuda")
    mag = torch.zeros_like(ref)
    for k, lag in enumerate(lags):
        if 0 <= lag < nsep:
            q = x[:, :nsep - lag] * x[:, lag:]
            q = q if power else q.sign() * q.abs().sqrt()
            ref[:, k], mag[:, k] = q.sum(1), q.abs().sum(1)
    if sumlags:
        ref, mag = ref.sum(1), mag.sum(1)
    assert bool(((out.double() - ref).abs() <= 100 * 2.0 ** -24 * mag).all())


@pytest.mark.parametrize("ntx,frames", [(2, 1), (13, 2)])
def test_channel_gradient_in_any_pixel_order(ntx, frames):
    """Parts whose taps span a long record (several segments of rows, pixels in random
    order) and parts of similar depth give the same channel gradient, up to the
    rounding of sums of some hundred terms in another order (float32: 1e-5)."""
    from pycbf_gb300 import adjoint
    r = np.random.default_rng(9)
    nrx, npx, nt, dt = 6, 5000, 2100, 4e-8
    depth = np.linspace(0.02, 0.7, npx) * nt * dt
    tabs = [depth[None] + r.uniform(0, 40, (ntx, 1)) * dt, 0.4 * depth[None] + r.uniform(0, 90, (nrx, 1)) * dt,
            np.ones((ntx, npx)), r.choice([0.0, 0.3, 1.0], (nrx, npx))]
    tabs = [torch.as_tensor(t, dtype=torch.float32, device="cuda") for t in tabs]
    rf = torch.randn((frames, ntx, nrx, nt), device="cuda")
    gout = torch.randn((frames, npx), device="cuda")
    perm = torch.as_tensor(r.permutation(npx), device="cuda")
    got = []
    for order in (torch.arange(npx, device="cuda"), perm):
        x = rf.clone().requires_grad_(True)
        out = adjoint.das_tabbed(x, *[t[:, order].contiguous() for t in tabs], t0=0.0, dt=dt)
        out.backward(gout[:, order].contiguous())
        got.append(x.grad.double())
    assert float(got[0].abs().max()) > 0
    assert float((got[0] - got[1]).norm() / got[0].norm()) < 1e-5
