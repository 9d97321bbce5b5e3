"""Bins of more k-mers than a counting CTA's store holds against the oracle: short
minimizers, whose bins are split into key-hash parts, and a part that is too large after
all and comes back through the retry list."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

ACGT = np.frombuffer(b"ACGT", dtype=np.uint8)


def _same(got, want):
    got = got.sorted()
    order = np.lexsort(tuple(want.keys[:, i] for i in range(want.keys.shape[1])))
    assert np.array_equal(got.keys, want.keys[order]) and np.array_equal(got.counts, want.counts[order])


@pytest.mark.parametrize("k,m", [(15, 9), (27, 11), (40, 9)])
@pytest.mark.parametrize("copies,ci", [(1, 1), (8, 2)])
def test_short_minimizers(k, m, copies, ci):
    import tuna_gb300 as T
    rng = np.random.default_rng(100 * k + copies)
    g = rng.choice(ACGT, 2_000_000 // copies)
    seq = np.concatenate([np.roll(g, int(rng.integers(0, g.size))) for _ in range(copies)])
    seq[rng.integers(0, seq.size, 4_000)] = ord("N")
    with T.Context(0) as ctx:
        got, _ = ctx.run(k, m, seq=seq, ci=ci)
    want = O.count_stream(seq, k, m, ci=ci, threads=8)
    assert got.stats["heavy_groups"] > 0 and got.stats["distinct"] == want.stats["n_distinct"]
    _same(got, want)


def _core(m: int) -> np.ndarray:
    """A conserved m-mer with a small canonical hash: the minimizer of every k-mer over it."""
    rng = np.random.default_rng(5)
    return np.frombuffer(min((rng.choice(ACGT, m).tobytes() for _ in range(20_000)), key=O.nthash), dtype=np.uint8)


def test_part_that_comes_back():
    """5,800 records of 11 k-mers of one bin, half of them equal and half all different,
    the halves 40 Mbp apart, so that the records of one lie before the other's. The equal
    half first: few k-mers are seen before the store is full, the parts are too few for
    the rest, and what does not fit is counted by one launch more."""
    import tuna_gb300 as T
    k, m, half = 31, 21, 2_900
    rng = np.random.default_rng(7)
    rows = np.empty((2 * half, 102), dtype=np.uint8)
    rows[:, :40] = rng.choice(ACGT, (2 * half, 40))
    rows[:, 40:61] = _core(m)
    rows[:, 61:101] = rng.choice(ACGT, (2 * half, 40))
    rows[:, 101] = ord("N")
    rows[:half] = rows[0]
    same, other = rows[:half].ravel(), rows[half:].ravel()
    filler = np.append(np.tile(rng.choice(ACGT, 1_000_000), 40), np.uint8(ord("N")))
    launches = []
    with T.Context(0) as ctx:
        for seq in (np.concatenate([same, filler, other]), np.concatenate([other, filler, same])):
            got, _ = ctx.run(k, m, seq=seq)
            want = O.count_stream(seq, k, m, threads=8)
            # the equal records' other minimizers have large bins too, of few k-mers
            assert got.stats["heavy_groups"] >= 1 and got.stats["fallback_groups"] == 0
            _same(got, want)
            launches.append(got.stats["gpu_launches"])
    assert launches[0] == launches[1] + 1
