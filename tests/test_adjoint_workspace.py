"""The differentiable path's workspace (CPU: sizes only)."""
import pytest

from pycbf_gb300 import _lib, adjoint


@pytest.mark.parametrize("ntx,nrx", [(11, 128), (25, 1024)])
def test_delay_tables_are_paid_for_only_where_they_are_made(ntx, nrx):
    """Synthetic delay tables: for gradients of the channel data, up to 2^30 bytes."""
    L = _lib.load()
    info = _lib.RFInfo(ntx, nrx, 2, 0.0, 4e-8, 2048, 1, _lib.F32)
    row = 4 * (ntx + nrx)
    most = (1 << 30) // row
    for np_, made in ((1000, True), (most, True), (most + 1, False), (1 << 22, False)):
        plain = adjoint._workspace_bytes(L, info, np_, False)
        least = L.pycbf_gb_adjoint_workspace_bytes(info, np_)
        assert least + 8 * (ntx + nrx) * ((np_ + 127) // 128) <= plain <= 1.05 * least + 1e6
        assert adjoint._workspace_bytes(L, info, np_, True) - plain == (row * np_ if made else 0)


class _Stop(Exception):
    pass


@pytest.mark.parametrize("need_rf", [False, True])
def test_a_gradient_of_the_slowness_alone_asks_for_no_tables(need_rf, monkeypatch):
    import torch
    asked = []

    def workspace(L, info, np_, tables, device):
        asked.append(tables)
        raise _Stop
    monkeypatch.setattr(adjoint, "_workspace", workspace)

    class Ctx:
        saved_tensors = (torch.zeros(64, dtype=torch.uint8), torch.zeros(10))
        geom = (None, None)
        rf_meta = ((1, 2, 3, 16), torch.float32)
        spec = adjoint._Spec(0.0, 4e-8, 0.01, 3, 2)
        pixel_index = torch.zeros(10, dtype=torch.int32)
        needs_input_grad = (need_rf, True)
    with pytest.raises(_Stop):
        adjoint._SyntheticDAS.backward(Ctx, torch.zeros(1, 10))
    assert asked == [need_rf]
