"""The device planner's ways to share a batch out: several groups of warps over
the same matrices (small batches, also where the groups do not come out even),
one thread per matrix up to 1024, several in turn above.  FP32 SIMT is bit-exact
with the oracle whatever tiles are chosen, so the tolerance is zero, and a
matrix that the queue missed or held twice (beta = 1) shows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from gpu_util import make_batch, oracle_batch, assert_bits_equal  # noqa: E402
from test_framework_tc_gpu import run  # noqa: E402
import batchgemm_gb300 as bg  # noqa: E402


@pytest.mark.parametrize("n", [1, 31, 33, 97, 225, 352, 1024, 1025, 2100])
def test_every_matrix_once(cuda, n):
    rng = np.random.default_rng(n)
    M, N, K = (rng.integers(0, 41, n).tolist() for _ in range(3))
    for i in range(0, n, 50):  # the longest tiles, which step 0 finds
        M[i], N[i], K[i] = 200 + i % 7, 150, 300 - i % 11
    db, host = make_batch(M, N, K, seed=n)
    want = oracle_batch(db, host, 1.0, 1.0)
    for _ in range(2):
        db.C.copy_(torch.from_numpy(host[2]))
        run(db, M, N, K, 210, 300, "simt")
        torch.cuda.synchronize()
        bg.framework_check_device()
        assert_bits_equal(db.C.cpu().numpy(), want, "batch of %d" % n)
