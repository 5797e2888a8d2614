"""The SIMT planner's limit of 65535 tiles along M and along N, up to the
largest sizes an int holds: what is above it is refused, alone and beside
ordinary matrices."""
import ctypes

import pytest

INT_MAX = 2**31 - 1
LARGEST = 65535 * 128  # the longest tile side is 128


def items(lib, M, N, K):
    """Work items of the batch (-1: refused); the queue itself is not built."""
    ints = lambda v: (ctypes.c_int * len(v))(*v)
    return lib.bgemm_debug_simt_queue(ints(M), ints(N), ints(K), len(M), 304, -1, 1, None, None, 0)


@pytest.mark.parametrize("size", [INT_MAX, INT_MAX - 14, INT_MAX - 19, INT_MAX - 126,
                                  INT_MAX - 127, LARGEST + 1])
@pytest.mark.parametrize("other", [1, 8, 9, 20, 64, 128])
def test_above_the_limit_is_refused(built_lib, size, other):
    for m, n in ((size, other), (other, size), (size, size)):
        assert items(built_lib, [m], [n], [4]) == -1
        assert items(built_lib, [100, m, 30], [70, n, 30], [16, 4, 16]) == -1


@pytest.mark.parametrize("other", [1, 9, 128])
def test_the_limit_itself_is_planned(built_lib, other):
    assert items(built_lib, [LARGEST], [other], [4]) == 65535
    assert items(built_lib, [other], [LARGEST], [4]) == 65535
