"""A large drain's bytes, copied out by several threads: the bytes at the address, and the
same lines as the pairs."""
import ctypes
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest


@pytest.mark.parametrize("n", [1, 65535, 65536, 4 * 65536, 4 * 65536 + 1, (4 << 20) + 12345])
def test_copy_bytes(n):
    import tuna_gb300 as T
    src = np.random.default_rng(n).integers(0, 256, n, dtype=np.uint8)
    with ThreadPoolExecutor(T._COPY_THREADS) as pool:
        got = T._copy_bytes(src.ctypes.data, n, pool)
    assert got == src.tobytes() == ctypes.string_at(src.ctypes.data, n)


@pytest.mark.gpu
def test_large_drain():
    import tuna_gb300 as T
    seq = np.frombuffer(b"ACGT", dtype=np.uint8)[np.random.default_rng(1).integers(0, 4, 400_000)]
    with T.Context(0) as ctx:
        r, _ = ctx.run(31, 21, seq=seq, drain=0)
        assert len(r.formatted) > T._COPY_MIN
        want = T.tsv_blob(r.keys, r.counts, 31)
    assert b"\n".join(sorted(r.formatted.splitlines())) + b"\n" == want
