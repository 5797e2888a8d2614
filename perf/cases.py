"""Performance cases of the variable-size batched SGEMM: what a user's program calls, and how.

A case is a batch of matrix products C_i <- alpha op(A_i) op(B_i) + beta C_i of one size
distribution, one numeric mode and one public entry point:

  plan            Plan(...) made once, one execute per pass
  oneshot         sgemm_vbatched / sgemm_vbatched_ex with host size arrays (the plan cache)
  stream          one Plan for several batches: update + execute per batch
  framework       framework_gemm: device size arrays, FP32 SIMT, C_i += A_i B_i
  framework_mode  framework_gemm_mode: the same in a tensor-core mode

The sizes of a case follow from the case alone (its ``shape_seed``), the values of its matrices
from the seed of :func:`prepare`.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import batchgemm_gb300 as bg
from batchgemm_gb300 import workloads

DEFAULTS = {
    "entry": "plan",       # see above
    "mode": "simt",        # "simt", "tf32", "tf32x3", "bf16x3"
    "dist": "uniform",     # how M, N and K are drawn, see _shapes
    "batch": 256,          # matrices (of each batch, for a stream: the largest)
    "batches": 1,          # batches of a stream
    "lo": 16, "hi": 256,   # range of M, N and K
    "shape_seed": 0,
    "alpha": 1.0, "beta": 0.0,
    "values": "uniform",   # "uniform" in [-1, 1) or "normal" N(0, 1)
    "layout": "col", "trans_a": False, "trans_b": False,
    "pad": 0,              # leading dimension beyond the extent that it spans
    "align": 4,            # floats: every matrix starts at a multiple of this
    "simt_below": 0,       # plan option: smaller matrices go to the SIMT kernel
}


def _case(name, **kw):
    return dict(DEFAULTS, name=name, **kw)


def listed():
    return [
        # the smallest call: a handful of little matrices, where launches and host work count
        _case("tiny_oneshot_simt", entry="oneshot", batch=16, lo=4, hi=32),
        # the plain FP32 batch of small matrices, as the drop-in computes it
        _case("plain_256_simt", batch=256, lo=16, hi=256),
        # the same batch on the tensor cores: a short pre-pass and a short GEMM
        _case("plain_256_tf32x3", mode="tf32x3", batch=256, lo=16, hi=256),
        # FP32 SIMT at scale, every size from thin to large, C read and written
        _case("scale_2048_simt", dist="log", batch=2048, lo=32, hi=1024, beta=0.5),
        # the benchmark's headline: many small and a few large matrices in split TF32
        _case("skewed_4000_tf32x3", mode="tf32x3", dist="skewed", batch=4000, lo=512, hi=2048,
              values="normal"),
        # grouped-GEMM shape: one common N and K, a long-tailed M, single-product TF32
        _case("uneven_m_128_tf32", mode="tf32", dist="zipf", batch=128, lo=1, hi=1024),
        # a stream of unlike batches through one plan, thin matrices on the SIMT kernel
        _case("stream_mixed_tf32x3", entry="stream", mode="tf32x3", dist="log", batch=1024,
              batches=4, lo=1, hi=4096, alpha=1.0, beta=1.0, simt_below=64),
        # the reference framework's own call on its own shape file
        _case("framework_ref_256", entry="framework", dist="ref", batch=256, lo=16, hi=512,
              beta=1.0),
        # the same call with device sizes on the tensor cores, a skewed batch
        _case("framework_mode_tf32x3", entry="framework_mode", mode="tf32x3", dist="skewed",
              batch=1000, lo=512, hi=1536, beta=1.0),
        # row-major activations times transposed weights, odd sizes, padded rows, no alignment
        _case("row_nt_odd_bf16x3", entry="oneshot", mode="bf16x3", batch=96, lo=97, hi=1501,
              layout="row", trans_b=True, pad=3, align=1, alpha=0.5, beta=1.0),
        # A transposed in FP32 SIMT (the gradient of a weight), padded columns
        _case("tn_padded_simt", batch=512, lo=8, hi=300, trans_a=True, pad=5, align=1,
              alpha=-1.0, beta=1.0),
    ]


# A drawn case's useful flops stay below what the largest listed cases cost in the same mode.
_MOST_FLOPS = {"simt": 1.5e11, "tf32": 1.0e12, "tf32x3": 1.0e12, "bf16x3": 1.0e12}
_MOST_BYTES = 4.0e9


def _log_int(rng, lo, hi):
    return min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))


def draw(rng):
    c = dict(DEFAULTS)
    c["entry"] = rng.choice(["plan", "plan", "oneshot", "stream", "framework", "framework_mode"])
    c["mode"] = rng.choice(["simt", "tf32x3", "tf32x3", "tf32", "bf16x3"])
    c["dist"] = rng.choice(["uniform", "log", "skewed", "zipf"])
    c["batch"] = _log_int(rng, 1, 4096)
    c["hi"] = _log_int(rng, 24, 2048)
    c["lo"] = _log_int(rng, 1, max(1, c["hi"] // 2))
    c["shape_seed"] = rng.randrange(1 << 20)
    c["values"] = rng.choice(["uniform", "normal"])
    if c["entry"] in ("framework", "framework_mode"):
        c["beta"] = 1.0
        if c["entry"] == "framework":
            c["mode"] = "simt"
        elif c["mode"] == "simt":
            c["mode"] = "tf32x3"
        c["hi"] = min(c["hi"], 1024)
        c["lo"] = min(c["lo"], c["hi"])
    else:
        c["alpha"], c["beta"] = rng.choice([(1.0, 0.0), (1.0, 0.0), (1.0, 1.0), (0.5, 1.0),
                                            (1.0, 0.5)])
        c["layout"] = rng.choice(["col", "col", "row"])
        c["trans_a"], c["trans_b"] = rng.choice([(False, False), (False, False), (True, False),
                                                 (False, True)])
        c["pad"] = rng.choice([0, 0, 0, 1, 4, 7])
        c["align"] = rng.choice([4, 4, 64, 1])
        if c["entry"] != "oneshot" and c["mode"] != "simt":
            c["simt_below"] = rng.choice([0, 0, 64])
        if c["entry"] == "stream":
            c["batches"] = rng.randint(2, 4)
            c["batch"] = min(c["batch"], 1024)
    while c["batch"] > 1:
        w = work(c)
        if w["flops"] <= _MOST_FLOPS[c["mode"]] and w["bytes"] <= _MOST_BYTES:
            break
        c["batch"] //= 2
    return c


def _shapes(case, which):
    """(M, N, K) lists of batch number ``which`` of the case."""
    rng = np.random.default_rng([case["shape_seed"], which])
    n, lo, hi, dist = case["batch"], case["lo"], case["hi"], case["dist"]
    if case["entry"] == "stream":  # the batches of a stream differ in length too
        n = int(rng.integers(max(1, n // 16), n + 1))
    if dist == "ref":
        w = workloads.ref_dataset(n)
        return w.M, w.N, w.K
    if dist == "log":
        s = np.exp(rng.uniform(np.log(lo), np.log(hi + 1), (n, 3)))
        s = np.clip(np.floor(s).astype(np.int64), lo, hi)
    elif dist == "skewed":  # nine in ten matrices at most 64, the rest in the range
        big = rng.random(n) < 0.10
        s = np.where(big[:, None], rng.integers(lo, hi + 1, (n, 3)),
                     rng.integers(min(8, hi), min(64, hi) + 1, (n, 3)))
    elif dist == "zipf":    # N = K = hi, M long-tailed
        s = np.full((n, 3), hi, np.int64)
        s[:, 0] = np.clip(rng.zipf(1.2, n), 1, 8 * hi)
    else:
        s = rng.integers(lo, hi + 1, (n, 3))
    return s[:, 0].tolist(), s[:, 1].tolist(), s[:, 2].tolist()


class _Batch:
    """One batch in device memory: flat A, B and C buffers, sizes and pointer arrays."""

    def __init__(self, case, which, gen):
        self.M, self.N, self.K = _shapes(case, which)
        self.row = case["layout"] == "row"
        dims = {
            "A": list(zip(self.K, self.M) if case["trans_a"] else zip(self.M, self.K)),
            "B": list(zip(self.N, self.K) if case["trans_b"] else zip(self.K, self.N)),
            "C": list(zip(self.M, self.N)),
        }
        self.dims, self.ld, self.off, self.buf, self.ptr = dims, {}, {}, {}, {}
        for x in "ABC":
            cur, off, ld = 0, [], []
            for r, c in dims[x]:
                line, lines = (c, r) if self.row else (r, c)
                cur = -(-cur // case["align"]) * case["align"]
                off.append(cur)
                ld.append(line + case["pad"])
                cur += ld[-1] * lines
            buf = torch.empty(cur, dtype=torch.float32, device="cuda")
            if case["values"] == "normal":
                buf.normal_(generator=gen)
            else:
                buf.uniform_(-1.0, 1.0, generator=gen)
            self.off[x], self.ld[x], self.buf[x] = off, ld, buf
            self.ptr[x] = torch.from_numpy(np.asarray(off, np.int64) * 4
                                           + buf.data_ptr()).cuda()

    def view(self, x, i, buf=None):
        ld = self.ld[x][i]
        return torch.as_strided(self.buf[x] if buf is None else buf, self.dims[x][i],
                                (ld, 1) if self.row else (1, ld), self.off[x][i])

    def sizes(self):
        return tuple(bg.int_array(v) for v in (self.M, self.N, self.K, self.ld["A"],
                                               self.ld["B"], self.ld["C"]))


def _batches(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    return [_Batch(case, b, gen) for b in range(case["batches"])]


def prepare(case, seed):
    batches = _batches(case, seed)
    sizes = [b.sizes() for b in batches]
    state = {"case": case, "batches": batches, "sizes": sizes}
    entry = case["entry"]
    if entry in ("plan", "stream"):
        opts = dict(layout=case["layout"], trans_a=case["trans_a"], trans_b=case["trans_b"],
                    simt_below=case["simt_below"])
        if entry == "stream":
            opts["capacity"] = bg.max_requirements(
                bg.plan_requirements(*s, mode=case["mode"], **opts) for s in sizes)
        state["plan"] = bg.Plan(*sizes[0], mode=case["mode"], **opts)
    elif entry in ("framework", "framework_mode"):
        b = batches[0]
        state["dev"] = [torch.tensor(v, dtype=torch.int32, device="cuda")
                        for v in (b.M, b.N, b.K)]
        state["max_dim"] = max(max(b.M), max(b.N))
        state["max_k"] = max(b.K)
        state["elems"] = sum((m + n) * k for m, n, k in zip(b.M, b.N, b.K))
    return state


def run(state):
    case, batches = state["case"], state["batches"]
    entry, mode = case["entry"], case["mode"]
    alpha, beta = case["alpha"], case["beta"]
    for b, s in zip(batches, state["sizes"]):
        pa, pb, pc = (b.ptr[x].data_ptr() for x in "ABC")
        if entry == "plan":
            state["plan"].execute(alpha, pa, pb, beta, pc)
        elif entry == "stream":
            state["plan"].update(*s)
            state["plan"].execute(alpha, pa, pb, beta, pc)
        elif entry == "oneshot":
            m, n, k, lda, ldb, ldc = s
            if case["layout"] == "col" and not case["trans_a"] and not case["trans_b"]:
                bg.sgemm_vbatched(m, n, k, alpha, pa, lda, pb, ldb, beta, pc, ldc, mode=mode)
            else:
                bg.sgemm_vbatched_ex(case["layout"], case["trans_a"], case["trans_b"], m, n, k,
                                     alpha, pa, lda, pb, ldb, beta, pc, ldc, mode=mode)
        else:
            dm, dn, dk = (v.data_ptr() for v in state["dev"])
            if entry == "framework":
                bg.framework_gemm(dm, dn, dk, pa, pb, pc, len(b.M), state["max_dim"])
            else:
                bg.framework_gemm_mode(dm, dn, dk, pa, pb, pc, len(b.M), state["max_dim"],
                                       state["max_k"], mode=mode,
                                       max_operand_elems=state["elems"])
    return [b.buf["C"] for b in batches]


def work(case):
    flops = elems = 0
    for which in range(case["batches"]):
        m, n, k = (np.asarray(v, np.float64) for v in _shapes(case, which))
        flops += float((2.0 * m * n * k).sum())
        elems += float((m * k + k * n + (2 if case["beta"] != 0 else 1) * m * n).sum())
    return {"bytes": 4.0 * elems, "flops": flops}


def exact(case, seed):
    out = []
    for b in _batches(case, seed):
        c = b.buf["C"].double()
        for i in range(len(b.M)):
            x, y = b.view("A", i).double(), b.view("B", i).double()
            x = x.t() if case["trans_a"] else x
            y = y.t() if case["trans_b"] else y
            v = b.view("C", i, c)
            p = torch.matmul(x, y).mul_(case["alpha"])
            if case["beta"] != 0:
                p.add_(v, alpha=case["beta"])
            v.copy_(p)
        out.append(c)
    return out
