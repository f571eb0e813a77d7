"""Where a routine changes kernels by size or form, neither side may be the slow
one: times of calls on the two sides, or of a call and a larger one, compared
with wide margins.  Each is the least of several replays of a graph of 20 calls."""
import numpy as np
import pytest

from clgpu_b200 import iclblas as B

pytestmark = pytest.mark.gpu


@pytest.fixture()
def us(handle, cuda):
    """us(call): device time of call(handle) in microseconds."""
    import torch
    s = torch.cuda.Stream()
    handle.set_stream(s)

    def measure(call, reps=20):
        with torch.cuda.stream(s):
            assert call(handle) == B.SUCCESS
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            for _ in range(reps):
                assert call(handle) == B.SUCCESS
        best = np.inf
        for _ in range(6):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            with torch.cuda.stream(s):
                a.record(s)
                g.replay()
                b.record(s)
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b) * 1e3 / reps)
        del g
        return best

    yield measure
    handle.set_stream(torch.cuda.current_stream())


def buf(n, cplx, cuda):
    import torch
    return torch.rand(n, dtype=torch.complex64 if cplx else torch.float32, device=cuda)


@pytest.mark.parametrize("cplx", [False, True])
def test_trsv_of_one_row(us, cuda, cplx):
    """A solve of one row is no 64-row inverse."""
    A, x = buf(64 * 65, cplx, cuda) + 1, buf(64, cplx, cuda)
    f = B.iclblasCtrsv if cplx else B.iclblasStrsv
    one, full = (us(lambda h: f(h, 1, 0, 0, n, A, 65, x, 1)) for n in (1, 64))
    assert one <= 0.5 * full


@pytest.mark.parametrize("inc,shift", [(1, 0), (1, 1), (2, 0), (17, 0)])
def test_reductions_of_short_vectors(us, cuda, inc, shift):
    """Half the elements never take much longer (one block or several)."""
    import torch
    big = 18000
    x, y = buf(big * inc + 4, False, cuda)[shift:], buf(big * inc + 4, False, cuda)[shift:]
    xc, yc = buf(big * inc + 4, True, cuda)[shift:], buf(big * inc + 4, True, cuda)[shift:]
    r, ri = torch.zeros(1, dtype=torch.complex64, device=cuda), torch.zeros(1, dtype=torch.int32, device=cuda)
    for call in (lambda h, n: B.iclblasSdot(h, n, x, inc, y, inc, r), lambda h, n: B.iclblasSasum(h, n, x, inc, r),
                 lambda h, n: B.iclblasIsamax(h, n, x, inc, ri), lambda h, n: B.iclblasCdotc(h, n, xc, inc, yc, inc, r),
                 lambda h, n: B.iclblasScnrm2(h, n, xc, inc, r), lambda h, n: B.iclblasIcamax(h, n, xc, inc, ri)):
        several = us(lambda h: call(h, big))
        for n in (2048, 4096, 8192, 12000, 16384):
            assert us(lambda h: call(h, n)) <= 1.3 * several, n


@pytest.mark.parametrize("cplx", [False, True])
def test_gemv_t_of_tall_and_of_short_columns(us, cuda, cplx):
    """Unaligned columns against aligned ones: a few tall ones, many short ones."""
    f = B.iclblasCgemv if cplx else B.iclblasSgemv
    for m, n, factor in ((1_000_000, 4, 2.0), (100_000, 33, 2.0), (4, 100_000, 1.3), (33, 100_000, 1.3)):
        A, x, y = buf((m + 4) * n, cplx, cuda), buf(m, cplx, cuda), buf(n, cplx, cuda)
        odd, aligned = (us(lambda h: f(h, 1, m, n, 1.0, A, lda, x, 1, 0.0, y, 1)) for lda in (m | 1, m + -m % 4))
        assert odd <= factor * aligned + 1, (m, n)


@pytest.mark.parametrize("n", [2600, 5036, 12000])
def test_gemv_t_of_a_nearly_full_batch(us, cuda, n):
    """Unaligned columns of almost two batches of loads (256 rows each) take no
    longer than those of two and a half."""
    A, x, y = buf(641 * n, False, cuda), buf(640, False, cuda), buf(n, False, cuda)
    t508, t640 = (us(lambda h: B.iclblasSgemv(h, 1, m, n, 1.0, A, m + 1, x, 1, 0.0, y, 1)) for m in (508, 640))
    assert t508 <= 1.15 * t640


def test_gemv_t_at_two_slices_a_column(us, cuda):
    """Unaligned complex columns just below two slices take no longer than
    those just above; ten matrices in turn, together larger than L2."""
    from itertools import cycle
    n, size = 1700, 2051 * 1700
    A, x, y = buf(10 * size, True, cuda), buf(2049, True, cuda), buf(n, True, cuda)

    def time(m):
        at = cycle(range(0, 10 * size, size))
        return us(lambda h: B.iclblasCgemv(h, 1, m, n, 1.0, A[next(at):], m + 2, x, 1, 0.0, y, 1))

    assert time(2047) <= 1.15 * time(2049)


@pytest.mark.parametrize("cplx", [False, True])
def test_gemv_n_of_few_columns(us, cuda, cplx):
    """One column more than a batch of 32 is no other slice."""
    f = B.iclblasCgemv if cplx else B.iclblasSgemv
    A, x, y = buf(3000 * 33, cplx, cuda), buf(33, cplx, cuda), buf(3000, cplx, cuda)
    t33, t32 = (us(lambda h: f(h, 0, 3000, n, 1.0, A, 3000, x, 1, 0.0, y, 1)) for n in (33, 32))
    assert t33 <= 1.35 * t32
