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


def test_table_given_back():
    """A table of 2^27 slots (1.6 GB) of one bin is not kept by the context."""
    import torch
    import tuna_gb300 as T
    seq = _satellite(40_000_000)
    with T.Context(0) as ctx:
        before = torch.cuda.mem_get_info()[0]
        for _ in range(2):
            got, _ = ctx.run(31, 21, seq=seq)
            assert got.stats["fallback_groups"] >= 1 and len(got) == 5
            assert before - torch.cuda.mem_get_info()[0] < 12 << 27


# 400,000 k-mers: 44 and 60 bytes each have to fit for one pass, the table takes 12.6 and 21 MB
@pytest.mark.parametrize("k,tight", [(31, 20 << 20), (63, 26 << 20)])
def test_table_under_a_budget(k, tight):
    """Large bins are counted without a table where the budget has no room for one."""
    import tuna_gb300 as T
    seq = _satellite(400_000)
    want = None
    for budget, table in ((0, True), (200 << 20, True), (tight, False)):
        with T.Context(0, hbm_budget=budget) as ctx:
            got, _ = ctx.run(k, 21, seq=seq)
        assert got.stats["heavy_groups"] >= 1 and got.stats["phase2_passes"] == 1
        assert (got.stats["fallback_groups"] > 0) == table
        got = got.sorted()
        if want is not None:
            assert np.array_equal(got.keys, want.keys) and np.array_equal(got.counts, want.counts)
        want = got
    assert len(want) == 5


def test_bin_of_2_32_kmers():
    """More k-mers of one bin than its counter holds: refused, in one run, of a shard, in
    passes and with the records in host memory."""
    import torch
    import tuna_gb300 as T
    if torch.cuda.mem_get_info()[0] < 200 << 30:
        pytest.skip("the pairs take 53 GB")
    seq = _satellite(4_400_000_000)
    for budget, kw in ((0, {}), (0, dict(shard=(1, 2))), (8 << 30, {}), (0, dict(spill=(1 << 33,)))):
        with T.Context(0, hbm_budget=budget) as ctx:
            with pytest.raises(T.GpuError, match=r"more than 2\^32"):
                ctx.run(31, 21, seq=seq, **kw)
