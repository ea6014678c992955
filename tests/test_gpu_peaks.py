"""The L1 microbenchmarks count the loads that run: both widths go through one data path of 128
bytes a clock and SM, so neither form may measure above the other's rate or that path's."""
from __future__ import annotations

import ctypes

import pytest

pytestmark = pytest.mark.gpu


def test_l1_loads_stay_within_the_data_path(cuda):
    import torch
    from fanbeamctrecon_tensorflowop_gb300 import _build
    _build.build()
    lib = ctypes.CDLL(str(_build.PEAKS_PATH))
    sms = torch.cuda.get_device_properties(cuda).multi_processor_count
    rates = []
    for fn in (lib.ctpk_l1_load, lib.ctpk_l1_load_v8):
        fn.argtypes = [ctypes.c_int, ctypes.c_int] + 2 * [ctypes.POINTER(ctypes.c_double)]
        gbs, ms = ctypes.c_double(), ctypes.c_double()
        for _ in range(3):
            assert fn(4, 1000, ctypes.byref(gbs), ctypes.byref(ms)) == 0
            rates.append(gbs.value)
    narrow, wide = max(rates[:3]), max(rates[3:])
    assert wide <= 1.1 * narrow
    assert max(narrow, wide) <= 1.02 * 128 * sms * 2.07  # at the highest clock, 2070 MHz
