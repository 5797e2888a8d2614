"""The FP32 SIMT kernel's thin tiles (8 x 128, 128 x 8) in every storage of
their long operand: rows that start on 16 bytes and anywhere (each alignment of
the first row and of the rows after it), K around the slices of 32 and their
four-k steps, both forms of the tile.  Bit-exact with the oracle; guard bands
hold NaN, so a read outside a matrix that reached a sum would show.

And their time, as a ratio within one run: rows that start anywhere against
rows on 16 bytes (1.3 measured; 1.9 where every float is a copy of its own), a
long operand stored the other way round against one that is not (1.0; 1.7)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

import batchgemm_gb300 as bg  # noqa: E402
from gpu_util import make_batch, oracle_batch, assert_bits_equal  # noqa: E402
from test_trans_gpu import Case  # noqa: E402

KS = [0, 1, 2, 3, 4, 5, 28, 29, 31, 32, 33, 35, 36, 61, 63, 64, 65, 97, 128, 131]
LONG = [1, 2, 31, 127, 128, 129, 130, 257]


def sizes(seed, thin_m):
    rng = np.random.default_rng(seed)
    n = 2 * len(KS)
    a = rng.choice([1, 2, 4, 5, 7, 8], n).tolist()
    b = rng.choice(LONG, n).tolist()
    return (a, b, KS * 2) if thin_m else (b, a, KS * 2)


@pytest.mark.parametrize("cfg", [8, 9])
@pytest.mark.parametrize("offset", [0, 1, 2, 3])
@pytest.mark.parametrize("pad", [0, 1, 2, 3, 4])
def test_every_alignment_bit_exact(cuda, cfg, offset, pad):
    M, N, K = sizes(offset, cfg == 8)
    ld = lambda v: [(x + 3) // 4 * 4 + pad for x in [max(y, 1) for y in v]]
    db, host = make_batch(M, N, K, ld(M), ld(K), ld(M), offset=offset, seed=pad)
    alpha, beta = [(1.0, 0.0), (1.0, 1.0), (-0.5, 2.0)][(offset + pad) % 3]
    want = oracle_batch(db, host, alpha, beta)
    with db.plan("simt", force_tile_config=cfg) as p:
        db.execute(p, alpha, beta)
        torch.cuda.synchronize()
    assert_bits_equal(db.C.cpu().numpy(), want, "cfg %d" % cfg)


@pytest.mark.parametrize("cfg", [2, 3, 4, 5, 6, 8, 9])
@pytest.mark.parametrize("layout", ["col", "row"])
@pytest.mark.parametrize("ta,tb", [("N", "N"), ("T", "N"), ("N", "T"), ("T", "T")])
def test_every_storage_bit_exact(cuda, cfg, layout, ta, tb):
    M, N, K = sizes(cfg, cfg == 8)
    if cfg < 8:
        M, N = M[:12] + [70] * 4, N[:12] + [130] * 4
        K = K[8:24]
    c = Case(layout, ta, tb, M, N, K, seed=cfg, pad=cfg % 4)
    pA, pB, pC = c.ptrs()
    alpha, beta = [(1.0, 1.0), (0.5, -1.5)][cfg % 2]
    with bg.Plan(M, N, K, c.lda, c.ldb, c.ldc, mode="simt", layout=layout, trans_a=ta,
                 trans_b=tb, force_tile_config=cfg) as p:
        p.execute(alpha, pA, pB, beta, pC)
        torch.cuda.synchronize()
    for i, (g, w) in enumerate(zip(c.result(), c.expected_f32(alpha, beta))):
        np.testing.assert_array_equal(np.ascontiguousarray(g).view(np.uint32),
                                      np.ascontiguousarray(w).view(np.uint32),
                                      err_msg="matrix %d (%d, %d, %d)" % (i, M[i], N[i], K[i]))


def test_time_of_odd_rows_and_of_transposes(cuda):
    n, long, k = 600, 1024, 512
    ms = {}
    for name, M, N, pad, ta in (("aligned", 8, long, 0, False), ("odd", 8, long, 1, False),
                                ("transposed", long, 8, 0, True)):
        ld = lambda v: v + pad
        a, b, c = (torch.empty(n * s, device="cuda").uniform_(-1, 1)
                   for s in (ld(k if ta else M) * (M if ta else k), ld(k) * N, ld(M) * N))
        ptr = [torch.arange(n, device="cuda") * (x.numel() // n * 4) + x.data_ptr()
               for x in (a, b, c)]
        with bg.Plan([M] * n, [N] * n, [k] * n, [ld(k if ta else M)] * n, [ld(k)] * n,
                     [ld(M)] * n, mode="simt", trans_a=ta) as p:
            run = lambda: p.execute(1.0, *(x.data_ptr() for x in ptr[:2]), 0.0, ptr[2].data_ptr())
            for _ in range(3):
                run()
            t = []
            for _ in range(9):
                e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
                e0.record()
                run()
                e1.record()
                e1.synchronize()
                t.append(e0.elapsed_time(e1))
            ms[name] = sorted(t)[4]
    assert ms["odd"] < 1.6 * ms["aligned"], ms
    assert ms["transposed"] < 1.35 * ms["aligned"], ms
