"""Which time axes' calls read a staging plan (CPU)."""
import pytest

from pycbf_gb300 import _lib


@pytest.mark.parametrize("kind", ["nearest", "linear", "cubic"])
@pytest.mark.parametrize("t0,dt,nt,ntx,used", [
    (0.0, 4e-8, 2048, 11, 0),       # an ordinary axis
    (1.0, 4e-8, 2056, 11, 1),       # float32 delays three samples apart, the last one rounded up
    (1.0, 4e-8, 2048, 11, 0),       # the last one rounded down
    (1.0, 4e-8, 2056, 13, 0),       # more transmits than a plan takes
    (1.0, 4e-8, 2047, 11, 0),       # windows that a bulk copy cannot start at
])
def test_plan_used(kind, t0, dt, nt, ntx, used):
    info = _lib.RFInfo(ntx, 128, 0, t0, dt, nt, 1, _lib.F32)
    if kind == "cubic" and nt == 2047:
        used = 1  # a record is 16 bytes
    assert _lib.load().pycbf_gb_tabbed_plan_used(info, _lib.INTERP[kind]) == used


def test_plan_used_refuses_quietly():
    L = _lib.load()
    good = _lib.RFInfo(11, 128, 0, 1.0, 4e-8, 2056, 1, _lib.F32)
    assert L.pycbf_gb_tabbed_plan_used(good, _lib.INTERP["cubic"]) == 1
    assert L.pycbf_gb_tabbed_plan_used(None, 0) == 0
    assert L.pycbf_gb_tabbed_plan_used(good, -1) == 0
    assert L.pycbf_gb_tabbed_plan_used(good, 3) in (0, 1)
    assert L.pycbf_gb_tabbed_plan_used(good, _lib.INTERP["cubic"] + 7) == 0
