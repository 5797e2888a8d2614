"""The autotuner's tile times are the tiles' own: no packing in them, none taken
off.  The committed table holds the times of these tiles without packing, so a
measurement of today is close to it; with the pre-pass estimated and subtracted
from a call whose packing overlaps the GEMM it was a fraction of it."""
import pytest

pytestmark = pytest.mark.gpu

import ctypes  # noqa: E402

import batchgemm_gb300 as bg  # noqa: E402
from batchgemm_gb300 import autotune  # noqa: E402


@pytest.mark.parametrize("mode,cfg", [("tf32", 8), ("tf32x3", 8), ("tf32x3", 10), ("bf16x3", 9)])
@pytest.mark.parametrize("K", [512, 2048])
def test_pair_tile_time_is_near_the_table(cuda, mode, cfg, K):
    a, b = ctypes.c_float(), ctypes.c_float()
    bg.lib().bgemm_debug_tile_cost(autotune.MODE_IDS[mode], cfg, ctypes.byref(a), ctypes.byref(b))
    t, _ = autotune.measure(mode, cfg, K, bg.device_info()["num_sms"] // 2)
    assert 0.75 < t / (a.value + b.value * K) < 1.35, (t, a.value + b.value * K)
