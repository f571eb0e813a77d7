"""Pageable host operands around the sizes at which their copies change form
(plain copy, ring of pinned chunks, bounce buffers): the call's results equal
numpy's bit for bit, the arrays around an operand stay untouched, and handles
in several threads share the pools."""
import threading

import numpy as np
import pytest

from clgpu_b200 import iclblas as B

pytestmark = pytest.mark.gpu
KIB, MIB = 1 << 10, 1 << 20


@pytest.mark.parametrize("nbytes", [4, 128 * KIB - 4, 128 * KIB, MIB - 4, MIB, MIB + 4, 4 * MIB, 5 * MIB + 12,
                                    16 * MIB - 4, 16 * MIB])
def test_sizes(handle, nbytes):
    n = nbytes // 4
    rng = np.random.default_rng(n)
    x = rng.uniform(-1, 1, n).astype(np.float32)
    buf = rng.uniform(-1, 1, n + 2).astype(np.float32)
    before, y = buf.copy(), buf[1:n + 1]
    assert B.iclblasScopy(handle, n, x, 1, y, 1) == B.SUCCESS
    assert np.array_equal(y, x)
    assert buf[0] == before[0] and buf[-1] == before[-1]
    assert B.iclblasSscal(handle, n, 0.5, y, 1) == B.SUCCESS  # in and out through one ring
    assert np.array_equal(y, x * np.float32(0.5))


def test_threads(cuda):
    bad = []

    def work(seed):
        rng = np.random.default_rng(seed)
        with B.Handle() as h:
            for n in (300_000, 40_000, 1_500_000, 700_001):
                x = rng.uniform(-1, 1, n).astype(np.float32)
                y = np.zeros(n, np.float32)
                if B.iclblasScopy(h, n, x, 1, y, 1) != B.SUCCESS or not np.array_equal(x, y):
                    bad.append((seed, n))

    threads = [threading.Thread(target=work, args=(s,)) for s in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
