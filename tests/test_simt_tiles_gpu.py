"""The FP32 SIMT kernel's warp and CTA tiles side by side in one queue.

A batch mixes sizes on both sides of every tile edge (16, 32, 128, the thin
sides of 8 and the slices of 16 and 32 k) with large matrices, so that CTAs
change between tiles that all their warps share and tiles of single warps, and
warps leave CTA tiles to one another.  FP32 SIMT is bit-exact with the oracle's
fma chain, so the tolerance is zero."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from gpu_util import make_batch, oracle_batch, assert_bits_equal  # noqa: E402
from test_trans_gpu import Case  # noqa: E402
import batchgemm_gb300 as bg  # noqa: E402

SIDES = [1, 4, 7, 8, 9, 15, 16, 17, 31, 32, 33, 48, 49, 64, 96, 97, 127, 128, 129, 160, 257]
KS = [0, 1, 3, 4, 15, 16, 17, 31, 32, 33, 47, 64, 65, 130]


def sizes(seed, n):
    rng = np.random.default_rng(seed)
    M, N = rng.choice(SIDES, n).tolist(), rng.choice(SIDES, n).tolist()
    K = rng.choice(KS, n).tolist()
    for i in range(0, n, 8):  # large ones between them
        M[i], N[i], K[i] = 300 + i, 270 + 2 * i, 200 + i
    return M, N, K


@pytest.mark.parametrize("pad", [0, 1])
@pytest.mark.parametrize("alpha,beta", [(1.0, 0.0), (1.0, 1.0), (-0.5, 2.0)])
def test_mixed_queue_bit_exact(cuda, pad, alpha, beta):
    M, N, K = sizes(3 + pad, 120)
    # pad 0: every leading dimension a multiple of 4 (16-byte copies and stores)
    up = (lambda v: (max(v, 1) + 3) // 4 * 4) if pad == 0 else (lambda v: v + 1)
    db, host = make_batch(M, N, K, [up(v) for v in M], [up(v) for v in K], [up(v) for v in M],
                          seed=pad)
    want = oracle_batch(db, host, alpha, beta)
    with db.plan("simt") as p:
        hist = p.info()["tile_config_hist"]
        assert hist[7] > 0 and hist[0] + hist[1] > 0, hist  # CTA and warp tiles
        for _ in range(3):  # the queue resets itself
            db.C.copy_(torch.from_numpy(host[2]))
            db.execute(p, alpha, beta)
            torch.cuda.synchronize()
            assert_bits_equal(db.C.cpu().numpy(), want, "mixed queue")


@pytest.mark.parametrize("ta,tb", [("T", "N"), ("N", "T"), ("T", "T")])
def test_mixed_queue_transposed_bit_exact(cuda, ta, tb):
    M, N, K = sizes(11, 40)
    c = Case("col", ta, tb, M, N, K, seed=2)
    pA, pB, pC = c.ptrs()
    with bg.Plan(M, N, K, c.lda, c.ldb, c.ldc, mode="simt", trans_a=ta, trans_b=tb) as p:
        p.execute(0.5, pA, pB, -1.5, pC)
        torch.cuda.synchronize()
    for i, (g, w) in enumerate(zip(c.result(), c.expected_f32(0.5, -1.5))):
        np.testing.assert_array_equal(np.ascontiguousarray(g).view(np.uint32),
                                      np.ascontiguousarray(w).view(np.uint32),
                                      err_msg="matrix %d (%d, %d, %d)" % (i, M[i], N[i], K[i]))
