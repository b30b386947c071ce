"""Calls of several host threads at once (GPU): the shared memory that one call asks of a
kernel does not take another's away, nor a later plan's an earlier one's.  The calls are
repeated from a few lines of C, so that they overlap whatever the interpreter does."""
import ctypes as ct
import os
import shutil
import subprocess
import threading

import numpy as np
import pytest
import torch

from pycbf_gb300 import _lib
from pycbf_gb300.batch import BatchBeamformer, BatchConfig
from test_gpu_rx import _channels, _tabbed

pytestmark = pytest.mark.gpu

# the parameters of pycbf_gb_das_tabbed and of pycbf_gb_das_tabbed_adjoint
DAS = ("const void *rf, const void *data, const float *tt, const float *at, const float *tr, "
       "const float *ar, long long np, const int *pi, int interp, float thresh, int sum, "
       "const void *plan, float *out, void *ws, size_t nws, void *stream",
       "rf, data, tt, at, tr, ar, np, pi, interp, thresh, sum, plan, out, ws, nws, stream")
ADJ = ("const void *rf, const void *coef, const float *tt, const float *at, const float *tr, "
       "const float *ar, long long np, const int *pi, float thresh, int sum, const float *g, "
       "float *grf, float *gt, float *gr, void *ws, size_t nws, void *stream",
       "rf, coef, tt, at, tr, ar, np, pi, thresh, sum, g, grf, gt, gr, ws, nws, stream")
SOURCE = "#include <stddef.h>\n" + "".join(
    f"int {name}(int n, int (*f)({decl}), {decl}) {{\n"
    f"    for (int k = 0; k < n; ++k) {{ int st = f({args}); if (st) return st; }}\n    return 0;\n}}\n"
    for name, (decl, args) in (("repeat_das", DAS), ("repeat_adj", ADJ)))


@pytest.fixture(scope="module")
def repeat(tmp_path_factory):
    cc = shutil.which("gcc") or shutil.which("cc")
    if cc is None:
        pytest.skip("no C compiler")
    d = tmp_path_factory.mktemp("repeat")
    src, so = os.path.join(d, "repeat.c"), os.path.join(d, "repeat.so")
    with open(src, "w") as fp:
        fp.write(SOURCE)
    subprocess.run([cc, "-O1", "-shared", "-fPIC", src, "-o", so], check=True)
    L, R = _lib.load(), ct.CDLL(so)
    for name, f in (("repeat_das", L.pycbf_gb_das_tabbed), ("repeat_adj", L.pycbf_gb_das_tabbed_adjoint)):
        getattr(R, name).argtypes = [ct.c_int, ct.c_void_p, *f.argtypes]

    def call(which, n, *args):
        f = L.pycbf_gb_das_tabbed if which == "repeat_das" else L.pycbf_gb_das_tabbed_adjoint
        return getattr(R, which)(n, ct.cast(f, ct.c_void_p), *args)
    return call


def _image(repeat, ntx, nt, kind="nearest", sumtype="tx_and_rx", frames=1, nrx=5, npx=40):
    bf = _tabbed(ntx, nrx, npx, nt, ntx, interp={"kind": kind}, stage_channels=False)
    rf = _channels(bf, 1, frames)
    info = bf._rfinfo(frames)
    ws = torch.empty(bf._lib.pycbf_gb_workspace_bytes(ct.byref(info), bf._interp_code), dtype=torch.uint8,
                     device="cuda")
    out = torch.empty(frames * ntx * npx, device="cuda")
    P, (tt, at, tr, ar), s = _lib.ptr, bf._tables, torch.cuda.Stream()
    keep = (bf, rf, info, ws, out, s)
    return keep, lambda n: repeat(
        "repeat_das", n, ct.byref(info), P(rf), P(tt), P(at), P(tr), P(ar), npx, P(bf._pixel_index),
        bf._interp_code, 0.01, _lib.SUMTYPE[sumtype], None, P(out), P(ws), ws.numel(), s.cuda_stream)


def _gradient(repeat, ntx, nt, nrx=3, npx=40):
    bf = _tabbed(ntx, nrx, npx, nt, ntx, pixel_order="natural")
    info = bf._rfinfo(1)
    coef = torch.zeros((ntx, nrx, nt, 4), device="cuda")
    g, grf, gt = torch.ones(npx, device="cuda"), torch.empty((ntx, nrx, nt), device="cuda"), \
        torch.empty((ntx, npx), device="cuda")
    ws = torch.empty(bf._lib.pycbf_gb_adjoint_workspace_bytes(ct.byref(info), npx), dtype=torch.uint8,
                     device="cuda")
    P, (tt, at, tr, ar), s = _lib.ptr, bf._tables, torch.cuda.Stream()
    keep = (bf, coef, g, grf, gt, ws, info, s)
    return keep, lambda n: repeat(
        "repeat_adj", n, ct.byref(info), P(coef), P(tt), P(at), P(tr), P(ar), npx, None, 0.01,
        _lib.SUMTYPE["tx_and_rx"], P(g), P(grf), P(gt), None, P(ws), ws.numel(), s.cuda_stream)


PAIRS = {
    "receives over warps": lambda r: (_image(r, 1, 64), _image(r, 454, 64)),
    "one receive": lambda r: (_image(r, 100, 64, nrx=1), _image(r, 454, 64, nrx=1)),
    "per-transmit sums": lambda r: (_image(r, 49, 64, sumtype="rx_only"), _image(r, 220, 64, sumtype="rx_only")),
    "record lengths": lambda r: (_image(r, 2, 64, "cubic"), _image(r, 2, 9000, "cubic")),
    "frames": lambda r: (_image(r, 1, 64, "cubic", frames=2), _image(r, 454, 64, "cubic", frames=2)),
    "record lengths of pairs": lambda r: (_image(r, 2, 64, "cubic", frames=2),
                                          _image(r, 2, 9000, "cubic", frames=2)),
    "gradients": lambda r: (_gradient(r, 2, 64), _gradient(r, 128, 9000)),
}


@pytest.mark.parametrize("name", list(PAIRS))
def test_two_sizes_in_two_threads(name, repeat):
    pair = PAIRS[name](repeat)
    torch.cuda.synchronize()
    status = {}

    def work(k, call):
        for _ in range(20):
            status[k] = status.get(k, 0) or call(200)

    threads = [threading.Thread(target=work, args=(k, call)) for k, (_, call) in enumerate(pair)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert status == {0: 0, 1: 0}


def test_a_batch_after_a_smaller_one_was_planned():
    """The queue's launches of a batch of long records and 200 transmits, before and after
    a batch that needs less shared memory is planned."""
    make = lambda ntx, nt: _tabbed(ntx, 3, 100, nt, 1)
    big, small = make(200, 9000), make(4, 64)
    frames = lambda bf: [_channels(bf, 3)]
    first = BatchBeamformer([big], config=BatchConfig(tx_chunk=0))
    want = first(frames(big))[0].clone()
    BatchBeamformer([small], config=BatchConfig(tx_chunk=0))(frames(small))
    first._run(first.config)
    torch.cuda.synchronize()
    assert torch.equal(first.outputs[0], want)
    np.testing.assert_array_equal(want.cpu().numpy(), big(frames(big)[0]).ravel())
