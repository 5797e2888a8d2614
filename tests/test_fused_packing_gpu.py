"""Operand packing inside the CTA-pair GEMM kernel.

Batches with more tiles than the pre-pass packs ahead (four per CTA pair), so
that the rest is packed by the GEMM kernel's own warps while it runs: every
storage order and transposition (each has its own load path), aligned and odd
leading dimensions, K around the 32-k chunks, matrices without K, and repeated
executes (the queues and strip counts reset themselves).  The bound is the
tensor-core modes' own: |c - c64| <= f u sqrt(K) (|alpha| sum|ab| + |beta c0|)
with u = 2^-24 and f = 32 (3xTF32), 2^-16 and 8 (3xBF16), 2^-11 and 4 (TF32)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

import batchgemm_gb300 as bg  # noqa: E402
from test_trans_gpu import BOUND  # noqa: E402


def check(mode, layout, ta, tb, pad, M, N, K, alpha, beta):
    n = len(M)
    gen = torch.Generator(device="cuda").manual_seed(7)

    def stored(rows, cols):
        """(buffer, offsets, leading dimensions, views of op-order matrices)"""
        ld = [max(c if layout == "row" else r, 1) + pad for r, c in zip(rows, cols)]
        off, cur = [], 0
        for r, c, l in zip(rows, cols, ld):
            cur = -(-cur // 4) * 4
            off.append(cur)
            cur += l * (r if layout == "row" else c)
        buf = torch.empty(max(cur, 4), device="cuda").uniform_(-1, 1, generator=gen)
        view = lambda b, i: torch.as_strided(b, (rows[i], cols[i]),
                                             (ld[i], 1) if layout == "row" else (1, ld[i]), off[i])
        ptr = torch.tensor([buf.data_ptr() + 4 * o for o in off], device="cuda")
        return buf, ptr, ld, view

    A, pA, lda, va = stored(K, M) if ta else stored(M, K)
    B, pB, ldb, vb = stored(N, K) if tb else stored(K, N)
    C, pC, ldc, vc = stored(M, N)
    c0 = C.clone()
    factor, unit = BOUND[mode]
    with bg.Plan(M, N, K, lda, ldb, ldc, mode=mode, layout=layout, trans_a=ta, trans_b=tb,
                 kernel_family="pair") as p:
        assert p.info()["num_tiles"] > 5 * p.info()["grid"] // 2  # some of it packed in the GEMM
        first = None
        for _ in range(2):
            C.copy_(c0)
            p.execute(alpha, pA.data_ptr(), pB.data_ptr(), beta, pC.data_ptr())
            p.check_device()
            if first is None:
                first = C.clone()
        assert torch.equal(first.view(torch.int32), C.view(torch.int32))
    want, bound = c0.double(), torch.zeros_like(c0, dtype=torch.float64)
    for i in range(n):
        a, b = va(A, i).double(), vb(B, i).double()
        a, b = (a.t() if ta else a), (b.t() if tb else b)
        w, c = vc(want, i), vc(bound, i)
        c.copy_(factor * unit * max(K[i], 1) ** 0.5 *
                (abs(alpha) * (a.abs() @ b.abs()) + abs(beta) * w.abs()))
        w.copy_(alpha * (a @ b) + beta * w)
    over = (C.double() - want).abs() > bound + 1e-30
    assert not bool(over.any()), int(over.sum())


def sizes(seed, n=420):
    rng = np.random.default_rng(seed)
    M = rng.choice([1, 31, 32, 33, 200, 257, 300], n).tolist()
    N = rng.choice([1, 32, 65, 129, 256, 270], n).tolist()
    K = rng.choice([0, 1, 3, 31, 32, 33, 64, 95, 96, 97, 130, 257], n).tolist()
    return M, N, K


@pytest.mark.parametrize("layout,ta,tb", [("col", False, False), ("col", True, False),
                                          ("col", False, True), ("row", True, True)])
@pytest.mark.parametrize("pad", [0, 1, 4])
def test_packing_in_the_gemm_3xtf32(cuda, layout, ta, tb, pad):
    M, N, K = sizes(pad)
    if pad == 4:  # 16-byte aligned rows
        M, N, K = ([(v + 3) // 4 * 4 for v in x] for x in (M, N, K))
    check("tf32x3", layout, ta, tb, pad, M, N, K, 1.0, 0.0)


@pytest.mark.parametrize("mode", ["tf32", "bf16x3", "tf32x3"])
def test_packing_in_the_gemm_modes(cuda, mode):
    check(mode, "col", False, False, 1, *sizes(5), alpha=-0.5, beta=1.0)


@pytest.mark.parametrize("mode", ["tf32", "bf16x3", "tf32x3"])
def test_packing_in_the_gemm_device_sizes(cuda, mode):
    """The device-size entry divides the packing on the device (C += A B)."""
    M, N, K = sizes(9)
    gen = torch.Generator(device="cuda").manual_seed(3)
    mats = [[torch.empty((c, r), device="cuda").uniform_(-1, 1, generator=gen).t()
             for r, c in zip(x, y)] for x, y in ((M, K), (K, N), (M, N))]
    c0 = [c.t().clone().t() for c in mats[2]]
    dev = [torch.tensor(v, dtype=torch.int32, device="cuda") for v in (M, N, K)]
    ptr = [torch.tensor([m.data_ptr() for m in x], device="cuda") for x in mats]
    factor, unit = BOUND[mode]
    for _ in range(2):
        for c, o in zip(mats[2], c0):
            c.copy_(o)
        bg.framework_gemm_mode(*(v.data_ptr() for v in dev), *(v.data_ptr() for v in ptr), len(M),
                               300, 257, mode=mode)
        bg.framework_check_device()
        for a, b, c, o, k in zip(*mats, c0, K):
            a, b, o = a.double(), b.double(), o.double()
            bound = factor * unit * max(k, 1) ** 0.5 * (a.abs() @ b.abs() + o.abs()) + 1e-30
            assert bool(((c.double() - (a @ b + o)).abs() <= bound).all())
