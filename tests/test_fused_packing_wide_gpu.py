"""Operand packing inside the CTA-pair GEMM kernel, k contiguous and long: the
8 x 128 chunks at their edges (rows around 8 and 32, K around 128 and the K of
256 from which they are used, beside shorter K in the same batch).  The bound
is that of test_fused_packing_gpu."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from test_fused_packing_gpu import check  # noqa: E402

ROWS = [769, 775, 776, 777, 800, 801, 831, 1023]
KS = [131, 255, 256, 257, 259, 383, 384, 385, 511, 515, 640]


@pytest.mark.parametrize("mode", ["tf32x3", "bf16x3", "tf32"])
@pytest.mark.parametrize("pad", [0, 1])
def test_long_contiguous_k(cuda, mode, pad):
    n = 66
    M = [ROWS[i % len(ROWS)] for i in range(n)]
    N = [ROWS[i * 3 % len(ROWS)] for i in range(n)]
    K = [KS[i % len(KS)] for i in range(n)]
    check(mode, "col", True, False, pad, M, N, K, 0.5, 1.0)
