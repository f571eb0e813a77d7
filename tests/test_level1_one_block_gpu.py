"""Reductions at the lengths where they go from one block to several, which
depend on the stride, the alignment and the type, against FP64."""
import numpy as np
import pytest

import oracle_lib as O
from clgpu_b200 import iclblas as B

pytestmark = pytest.mark.gpu
F = np.float32


@pytest.mark.parametrize("inc,shift", [(1, 0), (1, 1), (2, 0), (17, 0)])
@pytest.mark.parametrize("n", [1700, 1701, 3200, 3201, 3400, 3401, 6400, 6401, 8192, 8193, 10240, 10241, 16384, 16385])
def test_reductions(handle, cuda, n, inc, shift):
    import torch
    handle.set_stream(torch.cuda.current_stream())
    rng = np.random.default_rng(n + inc)
    for dtype in (np.float32, np.complex64):
        def vec():
            v = O.colmajor(n * inc + 4, 1, n * inc + 4, rng, dtype)
            return torch.from_numpy(v).to(cuda)[shift:], v[shift:][:n * inc:inc]
        (x, xv), (y, yv) = vec(), vec()
        wide = np.complex128 if dtype == np.complex64 else np.float64
        xw, yw = xv.astype(wide), yv.astype(wide)
        mag = np.abs(xw.real) + np.abs(xw.imag)
        r, ri = torch.zeros(1, device=cuda), torch.zeros(1, dtype=torch.int32, device=cuda)
        # FP64 sums: one rounding to FP32 of the result
        if dtype == np.float32:
            assert B.iclblasSdot(handle, n, x, inc, y, inc, r) == B.SUCCESS
            dot = r.item()
            assert B.iclblasSdotNoAlloc(handle, n, x, inc, y, inc, r) == B.SUCCESS
            assert r.item() == dot
            assert abs(dot - xw @ yw) <= 1e-6 * (np.abs(xw) @ np.abs(yw))
            calls = (B.iclblasSnrm2, B.iclblasSasum, B.iclblasIsamax)
        else:
            rc = torch.zeros(1, dtype=torch.complex64, device=cuda)
            for f, want in ((B.iclblasCdotu, xw @ yw), (B.iclblasCdotc, xw.conj() @ yw)):
                assert f(handle, n, x, inc, y, inc, rc) == B.SUCCESS
                assert abs(rc.item() - want) <= 1e-6 * (np.abs(xw) @ np.abs(yw))
            calls = (B.iclblasScnrm2, B.iclblasScasum, B.iclblasIcamax)
        assert calls[0](handle, n, x, inc, r) == B.SUCCESS
        assert abs(r.item() - np.linalg.norm(xw)) <= 1e-6 * np.linalg.norm(xw)
        assert calls[1](handle, n, x, inc, r) == B.SUCCESS
        assert abs(r.item() - mag.sum()) <= 1e-6 * mag.sum()
        assert calls[2](handle, n, x, inc, ri) == B.SUCCESS
        assert ri.item() == first_max(xv)


def first_max(v):
    """First index of the largest |re| + |im|, in FP32 as the routine compares."""
    m = np.abs(v.real) + np.abs(v.imag) if np.iscomplexobj(v) else np.abs(v)
    return int(np.argmax(m.astype(F)))
