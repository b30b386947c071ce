"""Gradients at the edges of their kernels' division of the work (GPU)."""
import numpy as np
import pytest
import torch

from oracle import adjoint_ref
from pycbf_gb300 import adjoint
from test_gpu_rx import DT, _channels, _synthetic, _tabbed

pytestmark = pytest.mark.gpu


def _rel(a, b):
    a, b = a.detach().double().cpu(), b.detach().double().cpu()
    return float(torch.linalg.norm(a - b) / torch.linalg.norm(b))


@pytest.mark.parametrize("step", [37, 5, 32])
def test_channel_gradient_from_parts_with_shifted_windows(step):
    """Four parts of 2048 pixels whose windows of samples overlap and begin `step` samples
    apart, so that a sample's place in the window differs from part to part: the sums
    over the parts against float64 autograd (at most 4000 taps a sample; 1e-5 as for the
    other channel gradients), and the same bits every time."""
    ntx, nrx, npx, nt, t0, dt = 2, 3, 8192, 301, 1.3e-7, 4e-8
    r = np.random.default_rng(step)
    at = np.arange(npx) // 2048 * step + r.uniform(3, 120, npx)
    f32 = lambda a: torch.as_tensor(np.asarray(a, np.float32))
    tautx = f32(t0 + dt * (at + r.uniform(0, 2, (ntx, 1))))
    taurx = f32(dt * r.uniform(0, 40, (nrx, 1)) + np.zeros((1, npx)))
    apodtx, apodrx = f32(r.uniform(0.2, 1, (ntx, npx))), f32(r.uniform(0.2, 1, (nrx, npx)))
    rf, g = f32(r.standard_normal((1, ntx, nrx, nt))), f32(r.standard_normal((1, npx)))

    def grad():
        x = rf.cuda().requires_grad_(True)
        out = adjoint.das_tabbed(x, tautx.cuda(), taurx.cuda(), apodtx.cuda(), apodrx.cuda(), t0=t0, dt=dt)
        return torch.autograd.grad(out, x, g.cuda())[0]

    x64 = rf.double().requires_grad_(True)
    ref = adjoint_ref.das_tabbed_ref(x64, *(t.double() for t in (tautx, taurx, apodtx, apodrx)), t0, dt)
    want = torch.autograd.grad(ref, x64, g.double())[0]
    got = grad()
    assert _rel(got, want) <= 1e-5
    for _ in range(20):
        assert torch.equal(grad(), got)


@pytest.mark.parametrize("nframes", [1, 2])
@pytest.mark.parametrize("dtype", ["float32", "float16"])
@pytest.mark.parametrize("make", [_tabbed, _synthetic])
def test_upstream_gradient_of_pixels_without_taps_is_not_used(make, dtype, nframes):
    """Receives that are masked, or whose taps all miss the record, leave exact zeros in
    the per-receive images; whatever the upstream gradient is there, NaN included, every
    gradient is the one that zeros there give, bit for bit."""
    ntx, nrx, npx, nt = 3, 21, 333, 301
    bf = make(ntx, nrx, npx, nt, 4)
    rf = _channels(bf, 8, nframes if nframes > 1 else 0, DT[dtype])
    slow = torch.full((npx,), 1 / 1500.0, device="cuda")
    if make is _synthetic:
        slow[::7] *= 1.6  # past the end of the record for the farther receives

    def grads(fill):
        x = rf.clone().requires_grad_(True)
        if make is _synthetic:
            leaves = [x, slow.clone().requires_grad_(True)]
            out = adjoint.das_synthetic_slowness(*leaves, bf, sumtype="tx_only")
        else:
            ttx, atx, trx, arx = bf._tables
            leaves = [x, ttx.clone().requires_grad_(True), trx.clone().requires_grad_(True)]
            out = adjoint.das_tabbed(*leaves, atx, arx, t0=bf.t0, dt=bf.dt, thresh=bf.thresh,
                                     sumtype="tx_only")
        g = torch.randn(out.shape, generator=torch.Generator().manual_seed(9)).cuda()
        empty = out == 0
        assert 0 < int(empty.sum()) < empty.numel()
        return torch.autograd.grad(out, leaves, torch.where(empty, torch.full_like(g, fill), g))

    for zero, nan, inf in zip(*(grads(v) for v in (0.0, float("nan"), float("inf")))):
        assert torch.equal(zero, nan) and torch.equal(zero, inf)
        assert float(zero.abs().max()) > 0


def test_channel_gradient_of_parts_of_4096_tiles():
    """64 parts of 4096 tiles of 128 pixels, whose list in shared memory leaves no room for
    the kernel's static part below the default limit.  The image is linear in the channel
    data v, so <image(v), g> = <v, gradient>: sums of 8192 float32 taps a sample and part, 64
    parts, and 64 samples give 4e-6 of |image| |g| / sqrt(pixels); 1e-4 allowed."""
    npx, nt, t0, dt = 64 * 4096 * 128, 64, 0.0, 4e-8
    gen = torch.Generator(device="cuda").manual_seed(10)
    u = lambda a, b: torch.empty((1, npx), device="cuda").uniform_(a, b, generator=gen)
    tautx, taurx, apodtx, apodrx = u(0, 40 * dt), u(0, 20 * dt), u(0.5, 1), u(0.5, 1)
    v = torch.randn((1, 1, nt), generator=gen, device="cuda").requires_grad_(True)
    out = adjoint.das_tabbed(v, tautx, taurx, apodtx, apodrx, t0=t0, dt=dt)
    g = torch.randn(out.shape, generator=gen, device="cuda")
    grad = torch.autograd.grad(out, v, g)[0].double()
    image, g, v = out.detach().double(), g.double(), v.detach().double()
    tol = 1e-4 * float(image.norm()) * float(g.norm()) / npx ** 0.5
    assert abs(float((image * g).sum()) - float((v * grad).sum())) <= tol


@pytest.mark.parametrize("nframes", [1, 2])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("sumtype", ["tx_only", "tx_and_rx"])
@pytest.mark.parametrize("ntx,nrx,npx", [(1, 1, 33), (5, 3, 300), (13, 4, 129), (75, 2, 64), (128, 4, 31), (12, 8, 65), (75, 5, 97)])
def test_delay_gradients_of_few_receives(nframes, dtype, sumtype, ntx, nrx, npx):
    """Up to eight receives go to kernels of fewer warps: their delay gradients against those
    of a call whose further receives have no weight.  A receive's own are the same bits, and
    up to four receives, one a warp, so are the transmits'; beyond, the receives' terms are
    added in another order: each sum of n terms is off by at most (n - 1) 2^-24 of the sum of
    their magnitudes, here those of single-receive calls."""
    nt, dt, more = 301, 4e-8, 9
    r = np.random.default_rng(ntx)
    cuda = lambda a: torch.as_tensor(np.asarray(a, np.float32)).cuda()
    taurx, apodrx = r.uniform(0, 140, (more, npx)) * dt, r.choice([0.0, 0.02, 1.0], (more, npx))
    apodrx[nrx:] = 0
    tautx, apodtx = r.uniform(-30, 200, (ntx, npx)) * dt, r.uniform(-1, 1, (ntx, npx))
    rf = cuda(r.standard_normal((nframes, ntx, more, nt))).to(DT[dtype])
    g = cuda(r.standard_normal((nframes, more, npx) if sumtype == "tx_only" else (nframes, npx)))

    def grads(a, b):
        leaves = [cuda(t).requires_grad_(True) for t in (tautx, taurx[a:b])]
        out = adjoint.das_tabbed(rf[:, :, a:b].contiguous(), *leaves, cuda(apodtx), cuda(apodrx[a:b]),
                                 t0=0.0, dt=dt, sumtype=sumtype)
        up = g[:, a:b].contiguous() if sumtype == "tx_only" else g
        return torch.autograd.grad(out, leaves, up.reshape(out.shape))

    (few_tx, few_rx), (tx, rx) = grads(0, nrx), grads(0, more)
    assert float(few_tx.abs().max()) > 0 and float(few_rx.abs().max()) > 0
    assert torch.equal(few_rx, rx[:nrx])
    bound = 0 if nrx <= 4 else 2 * (nrx - 1) * 2.0 ** -24 * sum(grads(k, k + 1)[0].abs() for k in range(nrx))
    assert bool(((few_tx - tx).abs() <= bound).all())
