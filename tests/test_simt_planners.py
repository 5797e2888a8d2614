"""The SIMT planners agree: the host planner (plans, one-shot entries) and the
device planner (its host replay) share one model and one rule, and choose the
same tile configuration for every matrix of a batch."""
import numpy as np
import pytest

from test_abi import simt_queue
from test_framework_planner import fw_simt_plan


@pytest.mark.parametrize("n,lo,hi", [(1, 1, 300), (5, 1, 2000), (60, 1, 400), (64, 8, 64),
                                     (300, 1, 4096), (700, 16, 1024)])
def test_host_and_device_planner_choose_alike(built_lib, n, lo, hi):
    rng = np.random.default_rng(n)
    for _ in range(3):
        M, N, K = (np.exp(rng.uniform(np.log(lo), np.log(hi + 1), n)).astype(int).clip(lo, hi)
                   .tolist() for _ in range(3))
        host, _ = simt_queue(M, N, K)
        dev, _, err = fw_simt_plan(M, N, K, 4096)
        assert err == 0 and host == list(dev)
