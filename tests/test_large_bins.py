"""One bin of a very large number of k-mers: a satellite between single Ns, so that many
cut CTAs have a share of it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _satellite(n, unit=b"ACGTT", every=50_000):
    s = np.tile(np.frombuffer(unit, dtype=np.uint8), n // len(unit) + 1)[:n].copy()
    s[every - 1::every] = ord("N")
    return s


def test_table_of_2_32_slots():
    """2^30 k-mers of one bin: the most slots that a global table can have."""
    import torch
    import tuna_gb300 as T
    k, n = 31, (1 << 30) + 2_000_000
    if torch.cuda.mem_get_info()[0] < 90 << 30:
        pytest.skip("the table takes 52 GB")
    seq = _satellite(n)
    with T.Context(0) as ctx:
        got, _ = ctx.run(k, 21, seq=seq)
    runs = np.diff(np.flatnonzero(np.concatenate([[True], seq == ord("N"), [True]]))) - 1
    kmers = int(np.maximum(runs - (k - 1), 0).sum())
    assert (1 << 30) <= got.stats["kmers"] == kmers < (1 << 31)
    assert got.stats["fallback_groups"] >= 1
    # every run but the last begins at the same place of the unit (50,000 is a multiple of five)
    assert len(got) == 5 and int(got.counts.astype(np.uint64).sum()) == kmers
    assert int(got.counts.max()) - int(got.counts.min()) <= len(runs)
