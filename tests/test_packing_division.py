"""How the planners divide the operand packing between the pre-pass kernel and
the CTA-pair GEMM kernel, without a GPU: the strips behind the head are exactly
those that the GEMM's tiles wait for, matrix by matrix (a count that does not
match would be read before it is packed, or waited for in vain), and the head
holds the tiles that the pairs start with.  Host planner and device planner."""
import ctypes

import numpy as np
import pytest

import batchgemm_gb300 as bg

from test_framework_planner import fw_plan
from test_tc_planner import MODES, tc_plan, tile_dims

CLUSTERS = 76
HEAD_TILES = 4


def division(M, N, K, mode, family=2, clusters=CLUSTERS):
    n = len(M)
    ints = lambda v: (ctypes.c_int * max(n, 1))(*v)
    jobs, head, wait = ctypes.c_int(), ctypes.c_int(), (ctypes.c_int * max(n, 1))()
    assert bg.lib().bgemm_debug_tc_division(ints(M), ints(N), ints(K), n, MODES[mode], family, 152,
                                            clusters, ctypes.byref(jobs), ctypes.byref(head),
                                            wait) == 0
    return jobs.value, head.value, list(wait)[:n]


def device_division(M, N, K, mode, max_dim, max_k, elems=0, clusters=CLUSTERS):
    n = len(M)
    ints = lambda v: (ctypes.c_int * max(n, 1))(*v)
    jobs, head, wait = ctypes.c_int(), ctypes.c_int(), (ctypes.c_int * max(n, 1))()
    assert bg.lib().bgemm_debug_framework_tc_division(
        ints(M), ints(N), ints(K), n, max_dim, max_k, ctypes.c_longlong(elems), MODES[mode],
        clusters, ctypes.byref(jobs), ctypes.byref(head), wait) == 0
    return jobs.value, head.value, list(wait)[:n]


def batches():
    rng = np.random.default_rng(3)
    log = lambda n, hi: np.exp(rng.uniform(0, np.log(hi), n)).astype(int).tolist()
    yield "few", log(20, 900), log(20, 900), log(20, 700)
    yield "many", log(900, 900), log(900, 900), log(900, 700)
    yield "one K", [300] * 500, [200] * 500, [256] * 500
    yield "two K", [300] * 500, [200] * 500, [256] * 250 + [31] * 250
    yield "empty ones", [0, 5, 300] * 200, [7, 0, 300] * 200, [9, 9, 0] * 100 + [9, 9, 77] * 100
    yield "one", [900], [900], [700]
    yield "none", [], [], []


def check(M, N, K, strips, jobs, head, wait):
    assert len(strips) == jobs and 0 <= head <= jobs
    late = [0] * len(M)
    for mat, _, _ in strips[head:]:
        late[mat] += 1
    assert late == wait
    assert not {m for m, _, _ in strips[:head]} & {m for m, _, _ in strips[head:]}


@pytest.mark.parametrize("mode", list(MODES))
@pytest.mark.parametrize("family", [1, 2])
def test_host_division(built_lib, mode, family):
    for name, M, N, K in batches():
        cfgs, items, _, strips, _, _ = tc_plan(M, N, K, mode, family)
        jobs, head, wait = division(M, N, K, mode, family)
        check(M, N, K, strips.tolist(), jobs, head, wait)
        if family == 1:
            assert head == jobs
        elif head < jobs:
            early = sum(1 for m, _, _ in items.tolist() if not wait[m])
            assert early >= HEAD_TILES * CLUSTERS, name
    assert division(*[[300] * 900, [300] * 900, [200] * 900], mode, 2)[1] < 900 * 20


@pytest.mark.parametrize("mode", list(MODES))
def test_device_division(built_lib, mode):
    fused = 0
    for name, M, N, K in batches():
        items, strips, _, _, _, err = fw_plan(M, N, K, 900, 700, mode)
        jobs, head, wait = device_division(M, N, K, mode, 900, 700)
        assert err == 0
        check(M, N, K, strips.tolist(), jobs, head, wait)
        fused += head < jobs
    assert fused >= 2  # "many" and "two K"; whole bins of K: one K is never divided
    M, N, K = [300] * 900, [300] * 900, [200] * 900
    assert device_division(M, N, K, mode, 900, 700, elems=1000)[:2] == (0, 0)  # does not fit
