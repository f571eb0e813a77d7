"""The work that programs have this library do, as measurable cases.

Twelve listed cases and a generator of further ones.  Every case goes through
the public ctypes binding (clgpu_b200.iclblas): device operands are torch CUDA
tensors on torch's current stream, host operands are numpy arrays.  Matrices
are column-major: a tensor of shape (columns, ld) holds element (i, j) at
[j, i].

Families, and what each stands for in use:

  level1  short device vectors: the vector part of an iterative solver's step
          (dot, copy, axpy, nrm2, scal, iamax, asum with device results), where
          launches and latency count
  sweep   long vectors and large matrix-vector products: the bandwidth-bound
          level-1/2 sweep (axpy, dot, nrm2, asum, iamax, gemv N and T,
          complex gemv N and C)
  gemv    matrix-vector products of ordinary and ragged sizes, both directions
          (N, then T or C), real and complex, any leading dimension
  trsv    one triangular solve with one right-hand side, real and complex
  gemm    matrix products, real and complex, in the plain FP32 mode and in the
          tensor-core modes
  hgemm   half-precision products of 1x1-convolution shapes (rows = batch x
          height x width)
  trsm    triangular solves with many right-hand sides: forward, and for real
          data the adjoint (dB and dA) too
  batched uneven batched triangular solves, forward and adjoint, through a plan
  host    one product on ordinary (pageable) host arrays: the call blocks and
          returns with the result in host memory
"""
import math

import numpy as np
import torch

from clgpu_b200 import iclblas as B

MODES = {
    "plain": B.MATH_PLAIN_FP32,
    "tf32": B.MATH_TF32,
    "bf16x3": B.MATH_BF16X3,
    "bf16x6": B.MATH_BF16X6,
}
OPS = {"N": B.OP_N, "T": B.OP_T, "C": B.OP_C}


def listed():
    return [
        # a solver's vector step on a small system; an odd length
        {"name": "level1-4099", "family": "level1", "n": 4099},
        # the bandwidth sweep at its full size
        {"name": "sweep-2^28", "family": "sweep", "n": 1 << 28, "s": 16384, "c": 8192},
        # a complex operator of ragged shape inside a larger array, applied both ways
        {"name": "cgemv-3001x1777", "family": "gemv", "complex": True, "m": 3001, "n": 1777, "lda": 3003, "trans": "C",
         "beta": 0.0},
        # the triangular-solve configuration's single right-hand side
        {"name": "strsv-16384", "family": "trsv", "complex": False, "n": 16384, "lda": 16384, "uplo": "lower",
         "trans": "N", "diag": "non-unit"},
        # a complex back substitution of ordinary, ragged size
        {"name": "ctrsv-3001", "family": "trsv", "complex": True, "n": 3001, "lda": 3001, "uplo": "upper",
         "trans": "C", "diag": "non-unit"},
        # the drop-in product: plain FP32, alpha and beta as in the first configuration
        {"name": "sgemm-512-plain", "family": "gemm", "complex": False, "mode": "plain", "ta": "N", "tb": "N",
         "m": 512, "n": 512, "k": 512, "pad": 0, "beta": 0.5},
        # an ordinary ragged product in the default mode
        {"name": "sgemm-2000x1500x3001-plain", "family": "gemm", "complex": False, "mode": "plain", "ta": "T",
         "tb": "N", "m": 2000, "n": 1500, "k": 3001, "pad": 1, "beta": 0.0},
        # the large product at FP32 accuracy on the tensor cores
        {"name": "sgemm-8192-bf16x6", "family": "gemm", "complex": False, "mode": "bf16x6", "ta": "N", "tb": "N",
         "m": 8192, "n": 8192, "k": 8192, "pad": 0, "beta": 0.0},
        # a 28x28 ResNet-50 layer, 512 -> 128 channels, batch 32
        {"name": "hgemm-28x28-512-128", "family": "hgemm", "ta": "N", "tb": "N", "m": 25088, "n": 128, "k": 512,
         "beta": 0.0},
        # the triangular-solve configuration, forward and adjoint
        {"name": "strsm-8192x4096-bf16x3", "family": "trsm", "complex": False, "mode": "bf16x3", "backward": True,
         "side": "left", "uplo": "lower", "trans": "N", "diag": "non-unit", "m": 8192, "n": 4096, "pad": 0},
        # the batched configuration at FP32 accuracy, forward and adjoint
        {"name": "batched-512-bf16x6", "family": "batched", "mode": "bf16x6", "batch": 512, "order": 1024,
         "nrhs": 256},
        # a caller of the original API: host arrays in, host array out
        {"name": "host-sgemm-1024x768x512", "family": "host", "m": 1024, "n": 768, "k": 512, "beta": 0.0},
    ]


def _log(rng, lo, hi):
    """A whole number in [lo, hi], spread evenly over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    fam = rng.choice(["level1", "sweep", "gemv", "trsv", "gemm", "gemm", "hgemm", "trsm", "batched", "host"])
    if fam == "level1":
        return {"family": fam, "n": _log(rng, 256, 262144)}
    if fam == "sweep":
        return {"family": fam, "n": _log(rng, 1 << 22, 1 << 28), "s": _log(rng, 4096, 16384),
                "c": _log(rng, 2048, 8192)}
    cplx = rng.random() < 0.4
    if fam == "gemv":
        m, n = _log(rng, 200, 10000), _log(rng, 200, 10000)
        return {"family": fam, "complex": cplx, "m": m, "n": n, "lda": m + rng.choice([0, 0, 1, 2, 5]),
                "trans": rng.choice(["T", "C"]), "beta": rng.choice([0.0, 0.0, 0.5])}
    if fam == "trsv":
        n = _log(rng, 256, 8192 if cplx else 16384)
        return {"family": fam, "complex": cplx, "n": n, "lda": n + rng.choice([0, 0, 1, 3]),
                "uplo": rng.choice(["lower", "upper"]), "trans": rng.choice(["N", "T", "C"]),
                "diag": rng.choice(["non-unit", "non-unit", "unit"])}
    if fam == "gemm":
        mode = rng.choice(["plain", "plain", "tf32", "bf16x3", "bf16x6"])
        top = (1400 if cplx else 3200) if mode == "plain" else (2600 if cplx else 5000)
        return {"family": fam, "complex": cplx, "mode": mode, "ta": rng.choice(["N", "T", "C"]),
                "tb": rng.choice(["N", "T"]), "m": _log(rng, 96, top), "n": _log(rng, 96, top),
                "k": _log(rng, 96, top), "pad": rng.choice([0, 0, 1, 4]), "beta": rng.choice([0.0, 0.0, 0.5])}
    if fam == "hgemm":
        # batch x height x width rows of a 1x1 convolution
        side = rng.choice([7, 14, 28, 56])
        return {"family": fam, "ta": "N", "tb": rng.choice(["N", "N", "T"]), "m": rng.randint(4, 32) * side * side,
                "n": rng.choice([64, 128, 256, 512, 1000]), "k": rng.choice([64, 128, 256, 512, 1024]),
                "beta": rng.choice([0.0, 0.0, 0.5])}
    if fam == "trsm":
        mode = rng.choice(["plain", "tf32", "bf16x3", "bf16x6"])
        top = {True: 2048, False: 4096}[cplx] if mode != "plain" else {True: 1024, False: 2048}[cplx]
        return {"family": fam, "complex": cplx, "mode": mode, "backward": not cplx and rng.random() < 0.5,
                "side": rng.choice(["left", "left", "right"]), "uplo": rng.choice(["lower", "upper"]),
                "trans": rng.choice(["N", "T", "C"]), "diag": rng.choice(["non-unit", "non-unit", "unit"]),
                "m": _log(rng, 256, top), "n": _log(rng, 128, top), "pad": rng.choice([0, 0, 1, 4])}
    if fam == "batched":
        mode = rng.choice(["plain", "tf32", "bf16x3", "bf16x6"])
        return {"family": fam, "mode": mode, "batch": _log(rng, 16, 256 if mode == "plain" else 512),
                "order": _log(rng, 128, 1024), "nrhs": _log(rng, 16, 256)}
    return {"family": "host", "m": _log(rng, 64, 1536), "n": _log(rng, 64, 1536), "k": _log(rng, 64, 1536),
            "beta": rng.choice([0.0, 0.0, 0.5])}


# ------------------------------------------------------------------ inputs

def _gen(seed, device="cuda"):
    return torch.Generator(device=device).manual_seed(seed)


def _uniform(g, *shape, cplx=False):
    """Uniform(-1, 1) entries; complex: real and imaginary parts."""
    shape = (*shape, 2) if cplx else shape
    t = torch.rand(shape, generator=g, device="cuda").mul_(2).sub_(1)
    return torch.view_as_complex(t) if cplx else t


def _triangular(g, order, ld, cplx=False):
    """Diagonal Uniform(1, 2), every other entry N(0, 1) / sqrt(order): the
    triangle that a call does not read holds other data, as in a packed
    factorisation."""
    shape = (order, ld, 2) if cplx else (order, ld)
    t = torch.randn(shape, generator=g, device="cuda").mul_(1.0 / math.sqrt(order * (2 if cplx else 1)))
    if cplx:
        t = torch.view_as_complex(t)
    t[:, :order].diagonal().copy_(torch.rand(order, generator=g, device="cuda").add_(1))
    return t


class _State:
    """What a program holds between calls; the handle (and plan) end with it."""

    def __init__(self, case, mode="plain"):
        self.case = case
        self.plan = None
        self.h = B.Handle()
        self.h.set_stream(torch.cuda.current_stream())
        self.h.set_math_mode(MODES[mode])

    def __del__(self):
        torch.cuda.synchronize()
        if self.plan is not None:
            self.plan.destroy()
        self.h.destroy()


def _sizes(case):
    """Instance orders and right-hand sides of a batched case: the sizes are
    part of the case, spread evenly over [32, order] x [1, nrhs]."""
    rng = np.random.default_rng(case["batch"] * 7919 + case["order"] * 31 + case["nrhs"])
    n = rng.integers(32, case["order"] + 1, case["batch"])
    r = rng.integers(1, case["nrhs"] + 1, case["batch"])
    return n.astype(np.int64), r.astype(np.int64)


def _offsets(counts):
    """Start of each instance in a flat array (multiples of 128 entries) and
    the array's length."""
    starts = np.zeros(len(counts) + 1, dtype=np.int64)
    np.cumsum((counts + 127) // 128 * 128, out=starts[1:])
    return starts[:-1], int(starts[-1])


def _pointers(flat, starts):
    return torch.from_numpy(flat.data_ptr() + 4 * starts).cuda()


def _batched_inputs(case, seed):
    """(A, B, G): flat device arrays of all instances."""
    n, r = _sizes(case)
    a0, alen = _offsets(n * n)
    b0, blen = _offsets(n * r)
    g = _gen(seed)
    A = torch.randn(alen, generator=g, device="cuda")
    rhs = torch.randn(blen, generator=g, device="cuda")
    grad = torch.randn(blen, generator=g, device="cuda")
    diag = torch.rand(int(n.sum()), generator=g, device="cuda").add_(1)
    at = 0
    for i in range(len(n)):
        k = int(n[i])
        t = A[int(a0[i]):int(a0[i]) + k * k].view(k, k)
        t.mul_(1.0 / math.sqrt(k))
        t.diagonal().copy_(diag[at:at + k])
        at += k
        end = int(b0[i]) + k * int(r[i])  # nothing between one instance's entries and the next's
        rhs[end:(end + 127) // 128 * 128].zero_()
        grad[end:(end + 127) // 128 * 128].zero_()
    return A, rhs, grad


def _gemm_shape(case):
    """Stored (columns, ld) of A, B and C."""
    m, n, k, pad = case["m"], case["n"], case["k"], case.get("pad", 0)
    ra, ca = (m, k) if case["ta"] == "N" else (k, m)
    rb, cb = (k, n) if case["tb"] == "N" else (n, k)
    return (ca, ra + pad), (cb, rb + pad), (n, m + pad)


def prepare(case, seed):
    fam = case["family"]
    s = _State(case, case.get("mode", "plain"))
    g = _gen(seed)
    if fam == "level1":
        n = case["n"]
        s.x, s.w = _uniform(g, n), _uniform(g, n)
        s.v = torch.empty_like(s.x)
        s.dot, s.nrm, s.asum = (torch.zeros(1, device="cuda") for _ in range(3))
        s.imax = torch.zeros(1, dtype=torch.int32, device="cuda")
    elif fam == "sweep":
        n, ns, nc = case["n"], case["s"], case["c"]
        s.x, s.y = _uniform(g, n), _uniform(g, n)
        s.A, s.u, s.yn, s.yt = _uniform(g, ns, ns), _uniform(g, ns), *(torch.zeros(ns, device="cuda") for _ in range(2))
        s.Ac, s.uc = _uniform(g, nc, nc, cplx=True), _uniform(g, nc, cplx=True)
        s.ycn, s.ycc = (torch.zeros(nc, dtype=torch.complex64, device="cuda") for _ in range(2))
        s.dot, s.nrm, s.asum = (torch.zeros(1, device="cuda") for _ in range(3))
        s.imax = torch.zeros(1, dtype=torch.int32, device="cuda")
    elif fam == "gemv":
        m, n, c = case["m"], case["n"], case["complex"]
        s.A = _uniform(g, n, case["lda"], cplx=c)
        s.x, s.xt = _uniform(g, n, cplx=c), _uniform(g, m, cplx=c)
        s.y, s.yt = _uniform(g, m, cplx=c), _uniform(g, n, cplx=c)
    elif fam == "trsv":
        n, c = case["n"], case["complex"]
        s.A = _triangular(g, n, case["lda"], c)
        s.b = _uniform(g, n, cplx=c)
        s.x = torch.empty_like(s.b)
    elif fam == "gemm":
        sa, sb, sc = _gemm_shape(case)
        s.A, s.B, s.C = (_uniform(g, *t, cplx=case["complex"]) for t in (sa, sb, sc))
    elif fam == "hgemm":
        sa, sb, sc = _gemm_shape(case)
        s.A, s.B, s.C = (_uniform(g, *t).half() for t in (sa, sb, sc))
    elif fam == "trsm":
        m, n, c, pad = case["m"], case["n"], case["complex"], case["pad"]
        order = m if case["side"] == "left" else n
        s.A = _triangular(g, order, order + pad, c)
        s.B = _uniform(g, n, m, cplx=c)
        s.X = torch.empty_like(s.B)
        if case["backward"]:
            s.G = torch.randn(n, m, generator=g, device="cuda")
            s.dB = torch.empty_like(s.G)
            s.dA = torch.zeros_like(s.A)
    elif fam == "batched":
        n, r = _sizes(case)
        a0, b0 = _offsets(n * n)[0], _offsets(n * r)[0]
        s.A, s.B, s.G = _batched_inputs(case, seed)
        s.X, s.dB, s.dA = torch.zeros_like(s.B), torch.zeros_like(s.B), torch.zeros_like(s.A)
        s.pA, s.pdA = _pointers(s.A, a0), _pointers(s.dA, a0)
        s.pX, s.pdB = _pointers(s.X, b0), _pointers(s.dB, b0)
        s.plan = B.BatchPlan(s.h, "trsm", side=B.SIDE_LEFT, uplo=B.FILL_LOWER, trans=B.OP_N, diag=B.DIAG_NON_UNIT,
                             m=n.tolist(), n=r.tolist(), lda=n.tolist(), ldb=n.tolist())
        s.plan.set_inverse_reuse(True)
    elif fam == "host":
        rng = np.random.default_rng(seed)
        m, n, k = case["m"], case["n"], case["k"]
        s.A, s.B, s.C = (rng.uniform(-1, 1, t).astype(np.float32) for t in ((k, m), (n, k), (n, m)))
    return s


# ------------------------------------------------------------------ one pass

_UPLO = {"lower": B.FILL_LOWER, "upper": B.FILL_UPPER}
_DIAG = {"unit": B.DIAG_UNIT, "non-unit": B.DIAG_NON_UNIT}
_SIDE = {"left": B.SIDE_LEFT, "right": B.SIDE_RIGHT}


def run(s):
    c, h = s.case, s.h
    return _RUN[c["family"]](s, c, h)


def _run_level1(s, c, h):
    n = c["n"]
    B.check(B.iclblasSdot(h, n, s.x, 1, s.w, 1, s.dot))
    B.check(B.iclblasScopy(h, n, s.w, 1, s.v, 1))
    B.check(B.iclblasSaxpy(h, n, -0.37, s.x, 1, s.v, 1))
    B.check(B.iclblasSnrm2(h, n, s.v, 1, s.nrm))
    B.check(B.iclblasSscal(h, n, 0.71, s.v, 1))
    B.check(B.iclblasIsamax(h, n, s.v, 1, s.imax))
    B.check(B.iclblasSasum(h, n, s.v, 1, s.asum))
    return {"v": s.v, "dot": s.dot, "nrm": s.nrm, "asum": s.asum, "imax": s.imax}


def _run_sweep(s, c, h):
    n, ns, nc = c["n"], c["s"], c["c"]
    B.check(B.iclblasSaxpy(h, n, 0.5, s.x, 1, s.y, 1))
    B.check(B.iclblasSdot(h, n, s.x, 1, s.y, 1, s.dot))
    B.check(B.iclblasSnrm2(h, n, s.x, 1, s.nrm))
    B.check(B.iclblasSasum(h, n, s.x, 1, s.asum))
    B.check(B.iclblasIsamax(h, n, s.x, 1, s.imax))
    B.check(B.iclblasSgemv(h, B.OP_N, ns, ns, 1.5, s.A, ns, s.u, 1, 0.5, s.yn, 1))
    B.check(B.iclblasSgemv(h, B.OP_T, ns, ns, 1.5, s.A, ns, s.u, 1, 0.5, s.yt, 1))
    B.check(B.iclblasCgemv(h, B.OP_N, nc, nc, 1.5, s.Ac, nc, s.uc, 1, 0.5, s.ycn, 1))
    B.check(B.iclblasCgemv(h, B.OP_C, nc, nc, 1.5, s.Ac, nc, s.uc, 1, 0.5, s.ycc, 1))
    return {"y": s.y, "dot": s.dot, "nrm": s.nrm, "asum": s.asum, "imax": s.imax, "yn": s.yn, "yt": s.yt,
            "ycn": s.ycn, "ycc": s.ycc}


def _run_gemv(s, c, h):
    fn = B.iclblasCgemv if c["complex"] else B.iclblasSgemv
    B.check(fn(h, B.OP_N, c["m"], c["n"], 1.5, s.A, c["lda"], s.x, 1, c["beta"], s.y, 1))
    B.check(fn(h, OPS[c["trans"]], c["m"], c["n"], 1.5, s.A, c["lda"], s.xt, 1, c["beta"], s.yt, 1))
    return {"y": s.y, "yt": s.yt}


def _run_trsv(s, c, h):
    copy, fn = (B.iclblasCcopy, B.iclblasCtrsv) if c["complex"] else (B.iclblasScopy, B.iclblasStrsv)
    B.check(copy(h, c["n"], s.b, 1, s.x, 1))
    B.check(fn(h, _UPLO[c["uplo"]], OPS[c["trans"]], _DIAG[c["diag"]], c["n"], s.A, c["lda"], s.x, 1))
    return s.x


def _run_gemm(s, c, h):
    fn = B.iclblasCgemm if c["complex"] else B.iclblasSgemm
    B.check(fn(h, OPS[c["ta"]], OPS[c["tb"]], c["m"], c["n"], c["k"], 1.5, s.A, s.A.shape[1], s.B, s.B.shape[1],
               c["beta"], s.C, s.C.shape[1]))
    return s.C


def _run_hgemm(s, c, h):
    B.check(B.iclblasHgemm(h, OPS[c["ta"]], OPS[c["tb"]], c["m"], c["n"], c["k"], 1.0, s.A, s.A.shape[1], s.B,
                           s.B.shape[1], c["beta"], s.C, s.C.shape[1]))
    return s.C


def _run_trsm(s, c, h):
    m, n, lda = c["m"], c["n"], s.A.shape[1]
    how = (_SIDE[c["side"]], _UPLO[c["uplo"]], OPS[c["trans"]], _DIAG[c["diag"]])
    copy, fn = (B.iclblasCcopy, B.iclblasCtrsm) if c["complex"] else (B.iclblasScopy, B.iclblasStrsm)
    B.check(copy(h, m * n, s.B, 1, s.X, 1))
    B.check(fn(h, *how, m, n, 1.0, s.A, lda, s.X, m))
    if not c["backward"]:
        return s.X
    B.check(copy(h, m * n, s.G, 1, s.dB, 1))
    B.check(B.iclblasStrsm_backward(h, *how, m, n, 1.0, s.A, lda, s.X, m, s.dB, m, s.dA, lda))
    return {"X": s.X, "dB": s.dB, "dA": s.dA}


def _run_batched(s, c, h):
    B.check(B.iclblasScopy(h, s.B.numel(), s.B, 1, s.X, 1))
    B.check(B.iclblasScopy(h, s.G.numel(), s.G, 1, s.dB, 1))
    B.check(B.iclblasStrsmBatchedUneven(h, s.plan, 1.0, s.pA, s.pX))
    B.check(B.iclblasStrsmBatchedUnevenBackward(h, s.plan, 1.0, s.pA, s.pX, s.pdB, s.pdA))
    return {"X": s.X, "dB": s.dB, "dA": s.dA}


def _run_host(s, c, h):
    m, n, k = c["m"], c["n"], c["k"]
    B.check(B.iclblasSgemm(h, B.OP_N, B.OP_N, m, n, k, 1.5, s.A, m, s.B, k, c["beta"], s.C, m))
    return s.C


_RUN = {"level1": _run_level1, "sweep": _run_sweep, "gemv": _run_gemv, "trsv": _run_trsv, "gemm": _run_gemm,
        "hgemm": _run_hgemm, "trsm": _run_trsm, "batched": _run_batched, "host": _run_host}


# ------------------------------------------------------------------ work

def work(case):
    """Bytes (every input read once, every output written once) and floating
    operations of one pass."""
    fam = case["family"]
    if fam == "level1":
        n = case["n"]
        return {"bytes": 4.0 * n * 3, "flops": 10.0 * n}
    if fam == "sweep":
        n, ns, nc = case["n"], case["s"], case["c"]
        return {"bytes": 12.0 * n + 8.0 * n + 3 * 4.0 * n + 2 * 4.0 * (ns * ns + 3 * ns)
                + 2 * 8.0 * (nc * nc + 3 * nc),
                "flops": 8.0 * n + 4.0 * ns * ns + 16.0 * nc * nc}
    if fam == "gemv":
        m, n, e, f = case["m"], case["n"], 8 if case["complex"] else 4, 4 if case["complex"] else 1
        return {"bytes": e * (2.0 * m * n + 2 * m + 2 * n), "flops": 4.0 * f * m * n}
    if fam == "trsv":
        n, e, f = case["n"], 8 if case["complex"] else 4, 4 if case["complex"] else 1
        return {"bytes": e * (n * (n + 1) / 2 + 2.0 * n), "flops": 1.0 * f * n * n}
    if fam in ("gemm", "hgemm", "host"):
        m, n, k = case["m"], case["n"], case["k"]
        cplx = case.get("complex", False)
        e, f = 2 if fam == "hgemm" else 8 if cplx else 4, 4 if cplx else 1
        return {"bytes": e * (1.0 * m * k + k * n + m * n * (2 if case["beta"] else 1)), "flops": 2.0 * f * m * n * k}
    if fam == "trsm":
        m, n, e, f = case["m"], case["n"], 8 if case["complex"] else 4, 4 if case["complex"] else 1
        o, r = (m, n) if case["side"] == "left" else (n, m)
        both = 3 if case["backward"] else 1
        byt = e * (o * o / 2.0 + 2.0 * m * n)
        return {"bytes": byt + (e * (o * o * 1.5 + 3.0 * m * n) if case["backward"] else 0),
                "flops": both * 1.0 * f * o * o * r}
    n, r = _sizes(case)
    a, b, w = float((n * n).sum()), float((n * r).sum()), float((n * n * r).sum())
    return {"bytes": 4 * (a / 2 + 2 * b) + 4 * (1.5 * a + 3 * b), "flops": 3 * w}


# ------------------------------------------------------------------ 64 bits

def _wide(t):
    return t.to(torch.complex128 if t.is_complex() else torch.float64)


def _op(M, op):
    return M if op == "N" else M.T if op == "T" else M.conj().T


def _tri(A, order, uplo, diag):
    """The triangle that a solve reads, as a full 64-bit matrix."""
    T = _wide(A[:, :order]).T
    T = torch.tril(T) if uplo == "lower" else torch.triu(T)
    if diag == "unit":
        T = T.clone()
        T.diagonal().fill_(1)
    return T.contiguous()


def _solve(T, uplo, op, rhs):
    low = (uplo == "lower") == (op == "N")
    return torch.linalg.solve_triangular(_op(T, op).resolve_conj(), rhs, upper=not low)


def exact(case, seed):
    fam = case["family"]
    s = prepare(case, seed)
    if fam == "level1":
        x, w = _wide(s.x), _wide(s.w)
        v = w - 0.37 * x
        return {"v": 0.71 * v, "dot": torch.dot(x, w).reshape(1), "nrm": v.norm().reshape(1),
                "asum": (0.71 * v).abs().sum().reshape(1), "imax": None}
    if fam == "sweep":
        x, y = _wide(s.x), _wide(s.y)
        y.add_(x, alpha=0.5)
        out = {"y": y, "dot": torch.dot(x, y).reshape(1), "nrm": x.norm().reshape(1),
               "asum": x.abs().sum().reshape(1), "imax": None}
        A, u = _wide(s.A), _wide(s.u)
        out |= {"yn": 1.5 * (A.T @ u), "yt": 1.5 * (A @ u)}
        del A
        A, u = _wide(s.Ac), _wide(s.uc)
        return out | {"ycn": 1.5 * (A.T @ u), "ycc": 1.5 * (A.conj() @ u)}
    if fam == "gemv":
        A = _wide(s.A[:, :case["m"]]).T
        return {"y": 1.5 * (A @ _wide(s.x)) + case["beta"] * _wide(s.y),
                "yt": 1.5 * (_op(A, case["trans"]) @ _wide(s.xt)) + case["beta"] * _wide(s.yt)}
    if fam == "trsv":
        T = _tri(s.A, case["n"], case["uplo"], case["diag"])
        return _solve(T, case["uplo"], case["trans"], _wide(s.b)[:, None])[:, 0]
    if fam in ("gemm", "hgemm"):
        m, n, k = case["m"], case["n"], case["k"]
        ra, rb = m if case["ta"] == "N" else k, k if case["tb"] == "N" else n
        A, Bm = _op(_wide(s.A[:, :ra]).T, case["ta"]), _op(_wide(s.B[:, :rb]).T, case["tb"])
        C = _wide(s.C)
        alpha = 1.5 if fam == "gemm" else 1.0
        C[:, :m] = (alpha * (A @ Bm)).T + case["beta"] * C[:, :m]
        return C
    if fam == "host":
        A, Bm, C = (torch.from_numpy(t).double().cuda() for t in (s.A, s.B, s.C))
        return (1.5 * (Bm @ A) + case["beta"] * C).cpu().numpy()
    if fam == "trsm":
        m, n = case["m"], case["n"]
        left, uplo, op = case["side"] == "left", case["uplo"], case["trans"]
        order = m if left else n
        T = _tri(s.A, order, uplo, case["diag"])
        back = {"N": "T", "T": "N", "C": "N"}[op]  # the adjoint is of real data

        def solve(op, M):  # M: (n, m), a column-major m x n matrix
            if left:
                return _solve(T, uplo, op, M.T).T
            # X op(T) = M  <=>  op(T)^T X^T = M^T, and M holds that transpose
            t = _op(T, op).T.resolve_conj().contiguous()
            return torch.linalg.solve_triangular(t, M, upper=(uplo == "lower") == (op == "N"))

        X = solve(op, _wide(s.B)).contiguous()
        if not case["backward"]:
            return X
        W = solve(back, _wide(s.G)).contiguous()
        d = -(W.T @ X) if left else -(X @ W.T)  # of op(T)
        d = d if op == "N" else d.T
        d = torch.tril(d) if uplo == "lower" else torch.triu(d)
        if case["diag"] == "unit":
            d = d - torch.diag(d.diagonal())
        dA = torch.zeros(s.dA.shape, dtype=torch.float64, device="cuda")
        dA[:, :order] = d.T
        return {"X": X, "dB": W, "dA": dA}
    n, r = _sizes(case)
    a0, b0 = _offsets(n * n)[0], _offsets(n * r)[0]
    X, W = torch.zeros(s.B.shape, dtype=torch.float64, device="cuda"), torch.zeros(
        s.B.shape, dtype=torch.float64, device="cuda")
    dA = torch.zeros(s.A.shape, dtype=torch.float64, device="cuda")
    for i in range(len(n)):
        k, q, a, b = int(n[i]), int(r[i]), int(a0[i]), int(b0[i])
        T = torch.tril(s.A[a:a + k * k].view(k, k).double().T)
        x = torch.linalg.solve_triangular(T, s.B[b:b + k * q].view(q, k).double().T, upper=False)
        w = torch.linalg.solve_triangular(T.T, s.G[b:b + k * q].view(q, k).double().T, upper=True)
        X[b:b + k * q] = x.T.reshape(-1)
        W[b:b + k * q] = w.T.reshape(-1)
        dA[a:a + k * k] = torch.tril(-(w @ x.T)).T.reshape(-1)
    return {"X": X, "dB": W, "dA": dA}
