"""The batch queue at the edges of its work items (GPU)."""
import numpy as np
import pytest

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
