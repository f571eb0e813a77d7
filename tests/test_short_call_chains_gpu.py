"""Chains of short calls, each reading what the launch before it wrote, with no
host synchronisation between them: on the legacy stream, on a stream of its own,
and replayed from a CUDA graph, over aligned, odd and strided operands.  The
same bits as with a synchronisation after every call are expected: launches may
start early, but read only finished results."""
import pytest

from clgpu_b200 import iclblas as B

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("where", ["legacy", "stream", "graph"])
@pytest.mark.parametrize("n,lda,inc", [(64, 64, 1), (301, 303, 1), (1536, 1537, 1), (1100, 1101, 2), (1024, 1024, 1)])
def test_chain(handle, cuda, n, lda, inc, where):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(n + inc)
    A = ((torch.rand(n, lda, generator=gen, device="cuda") * 2 - 1) / n ** 0.5).contiguous()
    v0 = torch.rand(n * inc, generator=gen, device="cuda")
    handle.set_math_mode(0)
    steps = 8

    def chain(v, w, r, M, sync):
        def done(status):
            assert status == B.SUCCESS
            if sync:
                assert handle.synchronize() == B.SUCCESS
        for i in range(steps):
            done(B.iclblasSgemv(handle, i % 2, n, n, 1.0, A, lda, v, inc, 0.0, w, inc))
            done(B.iclblasSaxpy(handle, n, 0.5, v, inc, w, inc))
            done(B.iclblasSscal(handle, n, 0.75, w, inc))
            done(B.iclblasSdot(handle, n, v, inc, w, inc, r[i:]))
            done(B.iclblasSgemm(handle, 0, 0, n, 1, n, 1.0, A, lda, w, n, 0.0, M[i], n))
            v, w = w, v

    def bufs():
        return v0.clone(), torch.zeros_like(v0), torch.zeros(steps, device="cuda"), torch.zeros(steps, n, device="cuda")

    want, got = bufs(), bufs()
    s = torch.cuda.current_stream() if where == "legacy" else torch.cuda.Stream()
    torch.cuda.synchronize()
    handle.set_stream(s)
    with torch.cuda.stream(s):
        chain(*want, True)
        if where == "graph":
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=s):
                chain(*got, False)
            for _ in range(3):
                got[0].copy_(v0)
                for t in got[1:]:
                    t.zero_()
                g.replay()
        else:
            chain(*got, False)
    torch.cuda.synchronize()
    for a, b in zip(got, want):
        assert torch.equal(a, b)


@pytest.mark.parametrize("mode", [B.MATH_PLAIN_FP32, B.MATH_BF16X3])
def test_after_copies_and_fills_in_a_graph(handle, cuda, mode):
    """Captured calls behind copy and fill nodes, and a solve that forks onto
    the handle's second stream."""
    import torch
    n, nrhs = 1536, 1024
    gen = torch.Generator(device="cuda").manual_seed(5)
    A = torch.rand(n, n, generator=gen, device="cuda") / n
    A.diagonal().add_(1.0)
    X0 = torch.rand(nrhs, n, generator=gen, device="cuda")
    handle.set_math_mode(mode)

    def run(X, C):
        X.copy_(X0)
        assert B.iclblasStrsm(handle, 0, 1, 0, 0, n, nrhs, 1.0, A, n, X, n) == B.SUCCESS
        C.zero_()
        assert B.iclblasSgemm(handle, 0, 0, n, nrhs, n, 1.0, A, n, X, n, 1.0, C, n) == B.SUCCESS
        X0b = X.clone()
        assert B.iclblasSscal(handle, X0b.numel(), 0.5, X0b, 1) == B.SUCCESS
        C.add_(X0b)

    want, got = [[torch.empty_like(X0) for _ in range(2)] for _ in range(2)]
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    handle.set_stream(s)
    with torch.cuda.stream(s):
        run(*want)
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            run(*got)
        for _ in range(2):
            for t in got:
                t.fill_(float("nan"))
            g.replay()
    torch.cuda.synchronize()
    for a, b in zip(got, want):
        assert torch.equal(a, b)


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("n,lda,inc", [(64, 64, 1), (301, 303, 1), (1100, 1101, 2), (1024, 1024, 1)])
def test_complex_chain(handle, cuda, n, lda, inc, graph):
    """The same of the complex routines."""
    import torch
    gen = torch.Generator(device="cuda").manual_seed(n + inc)

    def rand(*shape):
        return torch.view_as_complex(torch.rand(*shape, 2, generator=gen, device="cuda") * 2 - 1)

    A, v0 = rand(n, lda) / n ** 0.5, rand(n * inc)
    handle.set_math_mode(0)
    steps = 6

    def chain(v, w, r, q, M, sync):
        def done(status):
            assert status == B.SUCCESS
            if sync:
                assert handle.synchronize() == B.SUCCESS
        for i in range(steps):
            done(B.iclblasCgemv(handle, i % 3, n, n, 1.0, A, lda, v, inc, 0.0, w, inc))
            done(B.iclblasCaxpy(handle, n, 0.5j, v, inc, w, inc))
            done(B.iclblasCscal(handle, n, 0.75, w, inc))
            done(B.iclblasCdotc(handle, n, v, inc, w, inc, r[i:]))
            done(B.iclblasScnrm2(handle, n, w, inc, q[i:]))
            done(B.iclblasCgemm(handle, 2 * (i % 2), 0, n, 1, n, 1.0, A, lda, w, n, 0.0, M[i], n))
            v, w = w, v

    def bufs():
        return (v0.clone(), torch.zeros_like(v0), torch.zeros(steps, dtype=v0.dtype, device="cuda"),
                torch.zeros(steps, device="cuda"), torch.zeros(steps, n, dtype=v0.dtype, device="cuda"))

    want, got = bufs(), bufs()
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    handle.set_stream(s)
    with torch.cuda.stream(s):
        chain(*want, True)
        if graph:
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=s):
                chain(*got, False)
            for _ in range(3):
                got[0].copy_(v0)
                for t in got[1:]:
                    t.zero_()
                g.replay()
        else:
            chain(*got, False)
    torch.cuda.synchronize()
    for a, b in zip(got, want):
        assert torch.equal(a, b)
    handle.set_stream(torch.cuda.current_stream())
