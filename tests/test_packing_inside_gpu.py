"""Operands packed inside the CTA-pair GEMM kernel against the same operands
packed by the pre-pass kernel: the same bits of C, whoever packs.

Every storage of A and B (each has its own way into shared memory), leading
dimensions on 16 bytes and odd, K around the 32-k chunks, the 128-k ones and
their ring of four buffers, values that are infinite, NaN, subnormal or near
the largest; the planner's own division with the matrices that it leaves to the
GEMM named; a captured graph whose updates move the division; the device-size
entry with new sizes between replays; a wait for strips that never come."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

import batchgemm_gb300 as bg  # noqa: E402
from test_packing_division import device_division, division  # noqa: E402
from test_trans_gpu import BOUND  # noqa: E402

RULE, BEFORE, INSIDE = 0, 1, 2
STORAGES = [("col", False, False), ("col", True, False), ("col", False, True),
            ("col", True, True), ("row", False, False)]


class Operands:
    def __init__(self, M, N, K, layout="col", ta=False, tb=False, pad=0, specials=False):
        self.sizes, self.opts = (M, N, K), dict(layout=layout, trans_a=ta, trans_b=tb)
        gen = torch.Generator(device="cuda").manual_seed(11)

        def stored(rows, cols):
            line = rows if layout == "col" else cols
            lines = cols if layout == "col" else rows
            ld = [max(v, 1) + pad for v in line]
            off = np.concatenate([[0], np.cumsum([(l * c + 3) // 4 * 4
                                                  for l, c in zip(ld, lines)])])
            buf = torch.empty(int(off[-1]) + 4, device="cuda").uniform_(-1, 1, generator=gen)
            return buf, torch.tensor(buf.data_ptr() + 4 * off[:-1], device="cuda"), ld

        self.A, self.pA, lda = stored(K, M) if ta else stored(M, K)
        self.B, self.pB, ldb = stored(N, K) if tb else stored(K, N)
        self.C, self.pC, ldc = stored(M, N)
        self.ld = (lda, ldb, ldc)
        if specials:
            bits = [0x7f800000, 0xff800000, 0x7fc00000, 0x00000001, 0x807fffff, 0x00800000,
                    0x7f7fffff, 0xff7fffff, 0x7f7fe000, 0x7f7ff000, 0x80000000, 0x33800000]
            v = torch.tensor(np.array(bits, np.uint32).view(np.int32), device="cuda")
            for x in (self.A, self.B):
                at = torch.randint(x.numel(), (x.numel() // 400,), generator=gen, device="cuda")
                x.view(torch.int32)[at] = v[torch.arange(at.numel(), device="cuda") % len(bits)]
        self.C0 = self.C.clone()

    def plan(self, mode):
        return bg.Plan(*self.sizes, *self.ld, mode=mode, kernel_family="pair", **self.opts)

    def run(self, p, alpha=0.5, beta=1.0):
        self.C.copy_(self.C0)
        p.execute(alpha, self.pA.data_ptr(), self.pB.data_ptr(), beta, self.pC.data_ptr())
        p.check_device()
        return self.C.clone()

    def packed_by(self, p, who):
        assert bg.lib().bgemm_debug_plan_packing(p._h, who) == 0
        p.update(*self.sizes, *self.ld)
        return self.run(p)


def same(x, y):
    return bool(((x.view(torch.int32) == y.view(torch.int32)) | (x.isnan() & y.isnan())).all())


def sizes(n, ks, seed):
    rng = np.random.default_rng(seed)
    M = rng.choice([1, 31, 32, 33, 63, 130, 256, 257], n).tolist()
    N = rng.choice([1, 7, 8, 32, 65, 129, 256, 270], n).tolist()
    return M, N, [ks[i % len(ks)] for i in range(n)]


KS = [0, 1, 3, 31, 32, 33, 95, 96, 97, 127, 128, 129, 130, 255, 256, 257, 383, 384, 400, 515]


@pytest.mark.parametrize("mode", ["tf32", "tf32x3", "bf16x3"])
@pytest.mark.parametrize("layout,ta,tb", STORAGES)
@pytest.mark.parametrize("pad", [0, 1, 4])
def test_same_bits_whoever_packs(cuda, mode, layout, ta, tb, pad):
    M, N, K = sizes(120, KS, pad)
    if pad != 1:  # rows on 16 bytes
        M, N, K = ([(v + 3) // 4 * 4 for v in x] for x in (M, N, K))
    ops = Operands(M, N, K, layout, ta, tb, pad, specials=pad == 1)
    with ops.plan(mode) as p:
        before = ops.packed_by(p, BEFORE)
        for _ in range(2):  # the queues and counts reset themselves
            assert same(ops.packed_by(p, INSIDE), before)
        assert same(ops.packed_by(p, RULE), before)
    if pad != 1:
        assert bool(before.isfinite().all())


@pytest.mark.parametrize("mode", ["tf32", "tf32x3", "bf16x3"])
@pytest.mark.parametrize("ta", [False, True])
def test_the_rule_leaves_long_k_to_the_gemm(cuda, mode, ta):
    ks = [95, 96, 97, 130, 257, 383, 384, 400]
    M, N, K = sizes(160, ks, 5)
    M, N, K = M + [768] * 90, N + [768] * 90, K + [640] * 90
    ops = Operands(M, N, K, ta=ta, pad=1)
    with ops.plan(mode) as p:
        jobs, head, wait = division(M, N, K, mode, clusters=p.info()["grid"] // 2)
        late = {K[i] for i in range(160) if wait[i]}
        assert head < jobs and late >= {95, 96, 97, 130, 257}, (head, jobs, late)
        assert same(ops.run(p), ops.packed_by(p, BEFORE))


def bits_rne(x, drop):
    u = x.view(np.uint32).astype(np.uint64)
    return ((u + (1 << (drop - 1)) - 1 + ((u >> drop) & 1)) >> drop << drop).astype(
        np.uint32).view(np.float32)


@pytest.mark.parametrize("mode", ["tf32", "tf32x3", "bf16x3"])
@pytest.mark.parametrize("who", [BEFORE, INSIDE])
def test_rounding_of_every_bit_pattern(cuda, mode, who):
    """C = A * 1 with K = 1: the rounded operand itself (TF32), or the sum of
    its two parts, off by the second part's rounding and the accumulator's."""
    rng = np.random.default_rng(1)
    low = [0, 1, 0x0fff, 0x1000, 0x1001, 0x1fff, 0x2000, 0x3000, 0x7fff, 0x8000, 0x8001, 0xffff]
    u = np.concatenate([(np.arange(65536, dtype=np.uint32)[:, None] << 16
                         | np.array(low, np.uint32)).reshape(-1),
                        rng.integers(0, 1 << 32, 1 << 18, dtype=np.uint64).astype(np.uint32)])
    x = u.view(np.float32)
    top = np.float32(3.4e38) if mode == "tf32" else np.float32(2.0 ** 126)
    tiny = 2.0 ** -126 if mode == "tf32" else 2.0 ** -100
    x = np.ascontiguousarray(x[np.isfinite(x) & (np.abs(x) >= tiny) & (np.abs(x) <= top)])
    n = x.size // 4096
    x = x[:n * 4096]
    a = torch.from_numpy(x).cuda()
    b, c = torch.ones(n, device="cuda"), torch.zeros(n * 4096, device="cuda")
    ptr = [t.data_ptr() + 4 * s * torch.arange(n, device="cuda")
           for t, s in ((a, 4096), (b, 1), (c, 4096))]
    with bg.Plan([4096] * n, [1] * n, [1] * n, [4096] * n, [1] * n, [4096] * n, mode=mode,
                 kernel_family="pair") as p:
        assert bg.lib().bgemm_debug_plan_packing(p._h, who) == 0
        p.update([4096] * n, [1] * n, [1] * n, [4096] * n, [1] * n, [4096] * n)
        p.execute(1.0, ptr[0].data_ptr(), ptr[1].data_ptr(), 0.0, ptr[2].data_ptr())
        p.check_device()
    got = c.cpu().numpy()
    if mode == "tf32":
        assert np.array_equal(got.view(np.uint32), bits_rne(x, 13).view(np.uint32))
    else:
        off = np.abs(got.astype(np.float64) - x)
        assert (off <= np.abs(x) * (2.0 ** -22 if mode == "tf32x3" else 2.0 ** -17)).all()


@pytest.mark.parametrize("mode", ["tf32x3", "tf32"])
def test_updates_under_a_captured_graph_move_the_division(cuda, mode):
    big = lambda n, k: ([512] * n, [512] * n, [k] * n)
    batches = [sizes(60, KS, 1), tuple(x + y for x, y in zip(big(120, 600), sizes(200, KS, 2))),
               big(150, 130), tuple(x + y for x, y in zip(sizes(40, KS, 3), big(100, 515)))]
    all_ops = [Operands(*b) for b in batches]
    heads = []
    cap = bg.max_requirements(bg.plan_requirements(*o.sizes, *o.ld, mode=mode,
                                                   kernel_family="pair") for o in all_ops)
    n = cap["batch"]
    ptr = [torch.zeros(n, dtype=torch.int64, device="cuda") for _ in range(3)]
    s = torch.cuda.Stream()
    o = all_ops[0]
    with bg.Plan(*o.sizes, *o.ld, mode=mode, kernel_family="pair", capacity=cap, stream=s) as p:
        for t, q in zip(ptr, (o.pA, o.pB, o.pC)):
            t[:q.numel()] = q
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            p.execute(0.5, ptr[0].data_ptr(), ptr[1].data_ptr(), 1.0, ptr[2].data_ptr(), stream=s)
        for i in (0, 1, 2, 3, 1, 0):
            o = all_ops[i]
            jobs, head, _ = division(*o.sizes, mode, clusters=p.info()["grid"] // 2)
            heads.append((head, jobs))
            with torch.cuda.stream(s):
                for t, q in zip(ptr, (o.pA, o.pB, o.pC)):
                    t[:q.numel()] = q
                o.C.copy_(o.C0)
                p.update(*o.sizes, *o.ld, stream=s)
                g.replay()
            p.check_device(stream=s)
            got = o.C.clone()
            with o.plan(mode) as q:
                assert same(o.packed_by(q, BEFORE), got), i
    assert any(h == j for h, j in heads) and len({h for h, j in heads if h < j}) >= 2, heads


@pytest.mark.parametrize("mode", ["tf32x3", "bf16x3"])
def test_device_sizes_change_between_replays(cuda, mode):
    """Odd K that the device planner leaves to the GEMM (its strips counted by
    the host replay), other sizes in every replay of one captured call."""
    n, max_dim, max_k = 400, 300, 600
    rng = np.random.default_rng(4)
    batches = [(rng.integers(200, 301, n).tolist(), rng.integers(200, 301, n).tolist(),
                rng.choice(ks, n).tolist())
               for ks in ([600, 590, 97, 130, 257], [31, 33, 64], [601 - 1, 383, 129])]
    dev = [torch.zeros(n, dtype=torch.int32, device="cuda") for _ in range(3)]
    elems = max_dim * max(max_dim, max_k)
    buf = [torch.empty(n * elems, device="cuda").uniform_(-1, 1) for _ in range(2)]
    c = torch.zeros(n * max_dim * max_dim, device="cuda")
    ptr = [t.data_ptr() + 4 * e * torch.arange(n, device="cuda")
           for t, e in ((buf[0], elems), (buf[1], elems), (c, max_dim * max_dim))]
    s = torch.cuda.Stream()
    call = lambda: bg.framework_gemm_mode(*(v.data_ptr() for v in dev), *(v.data_ptr() for v in ptr),
                                          n, max_dim, max_k, mode=mode, stream=s)
    torch.cuda.synchronize()
    call()  # scratch and constants before the capture
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        call()
    factor, unit = BOUND[mode]
    fused = 0
    for i in (0, 1, 2, 0):
        M, N, K = batches[i]
        jobs, head, wait = device_division(M, N, K, mode, max_dim, max_k)
        fused += head < jobs and any(w and k % 32 for w, k in zip(wait, K))
        with torch.cuda.stream(s):
            for d, v in zip(dev, (M, N, K)):
                d.copy_(torch.tensor(v, dtype=torch.int32))
            c.fill_(0.25)
            g.replay()
        torch.cuda.synchronize()
        bg.framework_check_device()
        for j in range(0, n, 7):
            m, nn, k = M[j], N[j], K[j]
            a = buf[0][j * elems:j * elems + m * k].view(k, m).t().double()
            b = buf[1][j * elems:j * elems + k * nn].view(nn, k).t().double()
            got = c[j * max_dim ** 2:j * max_dim ** 2 + m * nn].view(nn, m).t().double()
            bound = factor * unit * k ** 0.5 * (a.abs() @ b.abs() + 0.25)
            assert bool(((got - (a @ b + 0.25)).abs() <= bound).all()), (i, j)
    assert fused >= 2
    bg.framework_release()


def test_wait_for_strips_that_never_come(cuda):
    L = bg.lib()
    L.bgemm_debug_packed_wait_selftest.argtypes = [ctypes.c_ulonglong] + \
        [ctypes.POINTER(ctypes.c_int)] * 3
    err, ret, ok = ctypes.c_int(-1), ctypes.c_int(-1), ctypes.c_int(-1)
    assert L.bgemm_debug_packed_wait_selftest(2_000_000, ctypes.byref(err), ctypes.byref(ret),
                                              ctypes.byref(ok)) == 0
    assert (err.value, ret.value, ok.value) == (1, 1, 0)
    torch.cuda.synchronize()  # the context is usable
