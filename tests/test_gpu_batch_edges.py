"""The batch queue at the edges of its work items (GPU)."""
import numpy as np
import pytest
import torch

from pycbf_gb300 import _lib
from pycbf_gb300.batch import BatchBeamformer, BatchConfig
from test_gpu_rx import _channels, _synthetic, _tabbed

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("make", [_tabbed, _synthetic])
@pytest.mark.parametrize("ntx", [13, 449, 450, 451, 452, 453])
def test_most_transmits_of_the_queue(make, ntx):
    """Transmit delays in a column of shared memory, up to the size whose padding no longer
    fits beside the queue's own part: the single-frame images, bit for bit."""
    bf = make(ntx, 9, 200, 301, ntx)
    rf = _channels(bf, 11)
    batch = BatchBeamformer([bf], config=BatchConfig(tx_chunk=0))
    got = batch([rf])[0].cpu().numpy()
    assert np.abs(got).max() > 0
    np.testing.assert_array_equal(got, bf(rf).ravel())


def test_one_transmit_more_is_refused_when_planned():
    """Not at the first run: the plan's own call."""
    with pytest.raises(_lib.GPUError, match="pycbf_gb_batch_plan"):
        BatchBeamformer([_tabbed(454, 2, 40, 64, 1)], config=BatchConfig(tx_chunk=0))


@pytest.mark.parametrize("storages", [("float32",), ("float16",), ("float32", "float16")])
def test_an_item_ends_with_its_job(storages):
    """Jobs of one tile in items of one and of eight tiles (a kernel of one storage type and
    that of several): the same work, so about the same time -- three times allowed, where
    eight tiles' worth would take eight."""
    bfs = [_tabbed(40, 64, 100, 301, 2, storage=storages[k % len(storages)]) for k in range(4)]
    frames = [_channels(bf, 12) for bf in bfs]
    us, images = [], []
    for tiles in (1, 8):
        batch = BatchBeamformer(bfs, config=BatchConfig(tx_chunk=0, tiles_per_item=tiles))
        images.append([o.clone() for o in batch(frames)])
        us.append(min(batch.time_config(batch.config, 20) for _ in range(5)))
    assert us[1] <= 3 * us[0]
    for a, b in zip(*images):
        assert torch.equal(a, b)
