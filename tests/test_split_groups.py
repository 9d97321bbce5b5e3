"""Bins of more k-mers than a CTA's store holds (few minimizers: a short m, whose hash has
few values), split into key-hash parts through global memory: the same pairs as the
path of a context with a memory budget, which takes no room for that."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _seq(n, copies, seed):
    rng = np.random.default_rng(seed)
    g = np.frombuffer(b"ACGT", dtype=np.uint8)[rng.integers(0, 4, n // copies)]
    s = np.concatenate([np.roll(g, int(rng.integers(0, g.size))) for _ in range(copies)])
    s[rng.integers(0, s.size, s.size // 500)] = ord("N")
    return s


# one copy: nearly all k-mers differ; eight: each k-mer about eight times. Below 4 MiB the
# groups are counted without a wait between the phases.
@pytest.mark.parametrize("k,m", [(15, 9), (27, 11), (40, 9)])
@pytest.mark.parametrize("n,copies,ci", [(2_000_000, 1, 1), (7_000_000, 1, 1), (7_000_000, 8, 2)])
def test_split_groups(k, m, n, copies, ci):
    import tuna_gb300 as T
    seq = _seq(n, copies, k + copies)
    with T.Context(0) as ctx, T.Context(0, hbm_budget=8 << 30) as plain:
        got, _ = ctx.run(k, m, seq=seq, ci=ci)
        want, _ = plain.run(k, m, seq=seq, ci=ci)
    assert got.stats["heavy_groups"] > 0 and got.stats["phase2_passes"] == want.stats["phase2_passes"]
    if ci == 1:
        assert int(got.counts.astype(np.uint64).sum()) == got.stats["kmers"]
    got, want = got.sorted(), want.sorted()
    assert np.array_equal(got.keys, want.keys) and np.array_equal(got.counts, want.counts)
