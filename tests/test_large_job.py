"""A job of more than 2^20 bins (whose descriptors have starts of 34 bits) and of more
groups than one k_recs launch places, against the same job's shards, which have 2^20
bins and one launch each."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [31, 63])
def test_against_shards(k):
    import tuna_gb300 as T
    rng = np.random.default_rng(k)
    g = np.frombuffer(b"ACGT", dtype=np.uint8)[rng.integers(0, 4, 1_200_000_000 // 4, dtype=np.uint8)]
    seq = np.concatenate([g] * 4)  # every k-mer four times, but for those at single Ns
    del g
    seq[5_000_000:8_000_000] = ord("A")
    seq[rng.integers(0, seq.size, 100_000)] = ord("N")
    with T.Context(0) as ctx:
        one, _ = ctx.run(k, 21, seq=seq, want_results=False, digest=True)
        shards = [ctx.run(k, 21, seq=seq, want_results=False, digest=True, shard=(s, 4))[0] for s in range(4)]
    # launches of k_recs: one for each 2^18 groups begun, of 4,096 or 3,072 k-mers
    per_launch = (4096 if k <= 31 else 3072) << 18
    assert one.stats["kmers"] >= per_launch and seq.size >= 1 << 29 and one.stats["phase2_passes"] == 1
    assert all(s.stats["out"] < per_launch for s in shards)
    assert one.digest["count_sum"] == one.stats["kmers"]
    for f in ("pairs", "count_sum"):
        assert one.digest[f] == sum(s.digest[f] for s in shards)
    for f in ("h1", "h2"):
        assert int(one.digest[f], 16) == sum(int(s.digest[f], 16) for s in shards) % (1 << 64)
