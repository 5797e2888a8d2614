"""The pre-pass's two ways through operands whose k is contiguous: rows on 16
bytes, and rows that start anywhere, which pass through shared memory.  The
packed operands must be the same bits, so the results are: no tolerance."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

import batchgemm_gb300 as bg  # noqa: E402

KS = [1, 2, 3, 4, 5, 31, 64, 127, 128, 129, 130, 131, 255, 256, 257, 259, 384, 515]
ROWS = [1, 3, 4, 5, 31, 32, 33, 64, 97]


def product(mode, M, N, K, values, pad):
    """C = op(A) B with A and B stored k-contiguous at leading dimension up4(K) + pad."""
    ld = [(k + 3) // 4 * 4 + pad for k in K]

    def stored(rows):
        off = np.concatenate([[0], np.cumsum([(r * l + 3) // 4 * 4 for r, l in zip(rows, ld)])])
        buf = torch.full((int(off[-1]),), float("nan"))
        for r, k, l, o in zip(rows, K, ld, off):
            torch.as_strided(buf, (r, k), (l, 1), int(o)).copy_(values(r, k))
        buf = buf.cuda()
        return buf, torch.tensor([buf.data_ptr() + 4 * int(o) for o in off[:-1]], device="cuda")

    A, pA = stored(M)
    B, pB = stored(N)
    offc = np.concatenate([[0], np.cumsum([(m * n + 3) // 4 * 4 for m, n in zip(M, N)])])
    C = torch.zeros(int(offc[-1]), device="cuda")
    pC = torch.tensor([C.data_ptr() + 4 * int(o) for o in offc[:-1]], device="cuda")
    with bg.Plan(M, N, K, ld, ld, M, mode=mode, trans_a=True) as p:
        p.execute(1.0, pA.data_ptr(), pB.data_ptr(), 0.0, pC.data_ptr())
        p.check_device()
    return C


@pytest.mark.parametrize("mode", ["tf32", "tf32x3", "bf16x3"])
def test_any_row_start_packs_the_same(cuda, mode):
    rng = np.random.default_rng(5)
    K = KS * 2
    M, N = rng.choice(ROWS, len(K)).tolist(), rng.choice(ROWS, len(K)).tolist()
    out = []
    for pad in (0, 1, 2, 3):
        gen = torch.Generator().manual_seed(9)
        out.append(product(mode, M, N, K, lambda r, k: torch.randn(r, k, generator=gen), pad))
    assert torch.isfinite(out[0]).all()
    for pad, c in enumerate(out):
        assert torch.equal(c.view(torch.int32), out[0].view(torch.int32)), "pad %d" % pad
