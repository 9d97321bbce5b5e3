"""Long files fed from host memory are copied and lexed in pieces of 16 MiB and more
(lex_append): the same stream as in one piece and as the oracle's parser, with
headers, lines and runs across piece boundaries and at the end-of-file rules."""
import re

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

MIB = 1 << 20
_RUN = re.compile(rb"[^ACGTacgt]+")


def _bases(n, seed):
    return np.frombuffer(b"ACGT", dtype=np.uint8)[np.random.default_rng(seed).integers(0, 4, n)]


def _fastq(total, seed, read=150):
    """About `total` bytes of reads of odd header lengths."""
    rng, out, size = np.random.default_rng(seed), [], 0
    seq = _bases(total, seed).tobytes()
    while size < total:
        h = b"@" + b"r" * int(rng.integers(0, 40)) + b"\n"
        ln = int(rng.integers(1, 2 * read))
        a = int(rng.integers(0, total - ln))
        rec = h + seq[a:a + ln] + b"\n+\n" + b"I" * ln + b"\n"
        out.append(rec)
        size += len(rec)
    return b"".join(out)


HEAD = b"@a\nACGTN" + b"\n+\nIIIII\n@b\n"


def _long_run(extra):
    """A FASTQ file that ends on a base of a sequence line begun two pieces before, `extra`
    bytes past a multiple of 64."""
    tail = _bases(40 * MIB, 2).tobytes()
    return HEAD + tail + b"A" * ((-len(HEAD) - len(tail)) % 64 + extra)


def _fasta():
    rows = np.full((40 * MIB // 61, 61), 10, dtype=np.uint8)
    rows[:, :60] = _bases(rows.shape[0] * 60, 3).reshape(-1, 60)
    return b">one\n" + rows.tobytes()


def _header_at(d):
    """A header that begins d bytes from the start of the second piece."""
    fa = _fasta()
    p = ((len(fa) + 1) // 2 + 16383) // 16384 * 16384 + d
    return fa[:p] + b">x y\n" + fa[p:]


CASES = {
    "fastq": lambda: _fastq(33 * MIB, 1),
    "fastq_dropped_run": lambda: _long_run(0),
    "fastq_kept_run": lambda: _long_run(1),
    "fasta": _fasta,
    "fasta_header_before": lambda: _header_at(-1),
    "fasta_header_at": lambda: _header_at(0),
    "fasta_header_long": lambda: b">a\nACGTA\n>" + b"h" * (35 * MIB) + b"\nACGTACGT\n",
}


@pytest.mark.parametrize("name", list(CASES))
def test_pieces(name):
    import tuna_gb300 as T
    data = CASES[name]()
    with T.Context(0) as ctx:
        got = ctx.lex(data)
    want = O.fastx_to_stream(data)
    assert [r for r in _RUN.split(got) if r] == [r for r in _RUN.split(want) if r]
