"""One minimizer's chain over nearly all of a stream: the cut CTA in whose chunk it
starts writes all of its records (a forced split every 256 - k positions), many more
than the other lists get."""
import ctypes

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _seq(unit, n, flank):
    from tuna_gb300 import synth
    s = np.tile(np.frombuffer(unit, dtype=np.uint8), n // len(unit) + 1)[:n].copy()
    s[:flank] = synth.genome(max(flank, 1), 5, 0.5)[:flank]
    return s


# up to 4 MiB the lists are sized before the records are counted, above it the cut runs
# again with lists as long as it found
@pytest.mark.parametrize("k,m", [(63, 21), (47, 31), (31, 12), (31, 21)])
@pytest.mark.parametrize("unit,n,flank", [(b"A", 4_000_000, 0), (b"ACGTT", 4 << 20, 200_000), (b"A", 4_600_000, 0),
                                          (b"ACGTT", 12_000_000, 100_000)])
def test_against_oracle(k, m, unit, n, flank):
    import tuna_gb300 as T
    seq = _seq(unit, n, flank)
    with T.Context(0) as ctx:
        got, _ = ctx.run(k, m, seq=seq)
    want = O.count_stream(seq, k, m, threads=8)
    assert int(got.counts.astype(np.uint64).sum()) == got.stats["kmers"] == n - k + 1
    got = got.sorted()
    order = np.lexsort(tuple(want.keys[:, i] for i in range(want.keys.shape[1])))
    assert np.array_equal(got.keys, want.keys[order]) and np.array_equal(got.counts, want.counts[order])


def test_pinned_input():
    """Phase 1 along with the copy, whose lists are too short here: again over the whole."""
    import tuna_gb300 as T
    L, n, k = T.library(), 34 << 20, 63
    with T.Context(0) as ctx, T.HostBuffer(n) as h_in, T.HostBuffer(16 * 16) as h_keys, T.HostBuffer(4 * 16) as h_cnt:
        h_in.array()[:] = ord("C")
        o = T._JobOpts(k, 21, 16, 1, (1 << 64) - 1, 0, 0)
        n_out = ctypes.c_uint64()
        st = T._Stats()
        rc = L.tg_count_seq(ctx.h, ctypes.byref(o), ctypes.c_void_p(h_in.ptr), n, ctypes.c_void_p(h_keys.ptr),
                            ctypes.c_void_p(h_cnt.ptr), 16, ctypes.byref(n_out), ctypes.byref(st))
        assert rc == 0, L.tg_last_error(ctx.h)
        assert n_out.value == 1 and st.distinct == 1
        assert int(h_cnt.array()[:4].view(np.uint32)[0]) == n - k + 1


def test_export():
    """The export cut's lists grow to what it found too; records [len][min_pos][bases]."""
    import tuna_gb300 as T
    n, k = 700_000, 63  # 3,627 records, in lists of 2,514 at first
    with T.Context(0) as ctx:
        got, parts = ctx.run(k, 21, seq=_seq(b"A", n, 0), n_parts=4, export=True)
    kmers = recs = 0
    for p in parts:
        at = 0
        while at < len(p):
            kmers += p[at] - (k - 1)
            recs += 1
            at += 2 + (p[at] + 3) // 4
    assert kmers == n - k + 1 and recs == got.stats["superkmers"]
