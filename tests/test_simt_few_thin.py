"""A few thin matrices of long K on the FP32 SIMT kernel: such a call ends with
its longest tile, and a 16 x 16 tile ends before a thin one (8 x 512 x 4096: 68
and 93 us).  Many of them fill the chip, and take the thin tiles that cost less
in all.  On the host, and by both planners alike."""
import pytest

from test_abi import simt_queue
from test_framework_planner import fw_simt_plan


@pytest.mark.parametrize("long", [512, 1000])
@pytest.mark.parametrize("k", [1024, 4096, 100000])
@pytest.mark.parametrize("thin_m", [True, False])
def test_few_take_small_tiles_and_many_thin_ones(built_lib, long, k, thin_m):
    for n, want in ((1, 0), (4, 0), (400, 8 if thin_m else 9)):
        M, N = ([8] * n, [long] * n) if thin_m else ([long] * n, [8] * n)
        host, _ = simt_queue(M, N, [k] * n)
        dev, _, err = fw_simt_plan(M, N, [k] * n, 4096)
        assert err == 0 and host == list(dev) == [want] * n, (n, k)
