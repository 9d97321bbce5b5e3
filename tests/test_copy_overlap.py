"""Phase 1 of a long page-locked stream or file runs piece by piece along with its copy
(P1Pipe): the same pairs as the job API, whose phase 1 runs over the whole stream,
with minimizer chains, runs of N and headers across tile and piece boundaries."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MIB = 1 << 20


def _bases(n, seed):
    """Copies of 2 Mbp, with one k-mer over many tiles, two k-mers in turn around the
    middle, a run of N and single Ns."""
    rng = np.random.default_rng(seed)
    g = np.frombuffer(b"ACGT", dtype=np.uint8)[rng.integers(0, 4, 2_000_003)]
    s = np.tile(g, n // g.size + 1)[:n].copy()
    s[n // 3:n // 3 + 3 * MIB] = ord("A")
    s[n // 2 - 40_000:n // 2 + 40_000] = np.tile(np.frombuffer(b"AT", dtype=np.uint8), 40_000)
    s[n // 5:n // 5 + 100_000] = ord("N")
    s[rng.integers(0, n, n // 5000)] = ord("N")
    return s


def _fasta(n):
    rows = np.full((n // 61, 61), 10, dtype=np.uint8)
    rows[:, :60] = _bases(rows.shape[0] * 60, 2).reshape(-1, 60)
    b = rows.tobytes()
    return np.frombuffer(b">one\n" + b[:n // 2] + b"\n>two\n" + b[n // 2:], dtype=np.uint8)


INPUTS = {"stream": lambda n: _bases(n, 1), "fasta": _fasta}


# the cut compiled for (31, 23), the generic one for one and for two key words
@pytest.mark.parametrize("kind,k,m", [("stream", 31, 23), ("stream", 31, 12), ("stream", 63, 21), ("fasta", 31, 23),
                                      ("fasta", 63, 21)])
@pytest.mark.parametrize("size", [32 * MIB, 40 * MIB + 13])
def test_overlapped_phase1(kind, k, m, size):
    import tuna_gb300 as T
    L = T.library()
    data = np.ascontiguousarray(INPUTS[kind](size))
    W = 1 if k <= 31 else 2
    with T.Context(0) as ctx:
        want, _ = ctx.run(k, m, **{"seq" if kind == "stream" else "fastx": data})
        want = want.sorted()
        n = len(want)
        with T.HostBuffer(data.size) as h_in, T.HostBuffer(8 * W * n) as h_keys, T.HostBuffer(4 * n) as h_cnt:
            h_in.array()[:] = data
            o = T._JobOpts(k, m, 16, 1, (1 << 64) - 1, 0, 0)
            n_out = ctypes.c_uint64()
            st = T._Stats()
            call = L.tg_count_seq if kind == "stream" else L.tg_count_fastx
            for _ in range(2):  # into new buffers, then into used ones
                rc = call(ctx.h, ctypes.byref(o), ctypes.c_void_p(h_in.ptr), data.size, ctypes.c_void_p(h_keys.ptr),
                          ctypes.c_void_p(h_cnt.ptr), n, ctypes.byref(n_out), ctypes.byref(st))
                assert rc == 0, L.tg_last_error(ctx.h)
                assert n_out.value == n
                got = T.Result(h_keys.array(np.uint64).reshape(n, W).copy(), h_cnt.array(np.uint32).copy(), {}, k).sorted()
                assert np.array_equal(got.keys, want.keys)
                assert np.array_equal(got.counts, want.counts)
                assert st.kmers == want.stats["kmers"] and st.superkmers == want.stats["superkmers"]


@pytest.mark.parametrize("k,m", [(31, 23), (63, 21)])
def test_overlapped_batch(k, m):
    """Samples of page-locked memory at odd addresses, an empty one and one of a base among them."""
    import tuna_gb300 as T
    L = T.library()
    W = 1 if k <= 31 else 2
    lens = [11 * MIB + 5, 0, 1, 20 * MIB + 17, 33, 9 * MIB]
    with T.Context(0) as ctx, T.HostBuffer(sum(lens) + 64 * len(lens)) as h_in:
        buf, at, smp = h_in.array(), 0, []
        for i, ln in enumerate(lens):
            at = (at + 15) // 16 * 16 + 3 * i
            buf[at:at + ln] = _bases(ln, i) if ln > 10 * MIB else _bases(11 * MIB, i)[:ln]
            smp.append(buf[at:at + ln])
            at += ln
        want, _ = ctx.run(k, m, samples=[s.copy() for s in smp])
        n = len(want)
        with T.HostBuffer(8 * W * n) as h_keys, T.HostBuffer(4 * n) as h_cnt:
            o = T._JobOpts(k, m, 16, 1, (1 << 64) - 1, 0, 0)
            n_out = ctypes.c_uint64()
            off = np.zeros(len(lens) + 1, dtype=np.uint64)
            ptrs = (ctypes.c_void_p * len(lens))(*[s.ctypes.data for s in smp])
            szs = (ctypes.c_size_t * len(lens))(*lens)
            rc = L.tg_count_batch(ctx.h, ctypes.byref(o), len(lens), ptrs, szs, ctypes.c_void_p(h_keys.ptr),
                                  ctypes.c_void_p(h_cnt.ptr), ctypes.c_void_p(off.ctypes.data), n, ctypes.byref(n_out),
                                  ctypes.byref(T._Stats()))
            assert rc == 0, L.tg_last_error(ctx.h)
            assert n_out.value == n and off[-1] == n
            keys, cnt = h_keys.array(np.uint64).reshape(n, W), h_cnt.array(np.uint32)
            for i in range(len(lens)):
                a, b = int(off[i]), int(off[i + 1])
                got = T.Result(keys[a:b].copy(), cnt[a:b].copy(), {}, k).sorted()
                w = want.sample(i).sorted()
                assert np.array_equal(got.keys, w.keys) and np.array_equal(got.counts, w.counts)
