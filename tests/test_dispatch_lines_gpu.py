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
