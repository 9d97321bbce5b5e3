"""Reads over a genome of a few long repeat families: bins with more k-mers than
a counting CTA's store holds (counted in rounds, as key-hash parts, or by many CTAs)
next to bins with none, on both sides of every size at which the path changes."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def reads():
    from tuna_gb300 import synth
    g = synth.genome(150_000, 5, 0.5, fam_a=(3, 1000, 0.8), div=(0.02, 0.02))
    return synth.fastq_sequence_stream(synth.reads_fastq(g, 20_000, 150, 0.005, 0.0, 9))


@pytest.mark.parametrize("k,m", [(63, 21), (47, 31), (33, 21), (31, 21), (31, 30), (25, 13), (21, 17), (9, 5)])
@pytest.mark.parametrize("ci", [1, 2])
def test_against_oracle(reads, k, m, ci):
    import tuna_gb300 as T
    with T.Context(0) as ctx:
        got, _ = ctx.run(k, m, seq=reads, ci=ci)
    want = O.count_stream(reads, k, m, ci=ci, threads=8)
    assert got.stats["distinct"] == want.stats["n_distinct"]
    assert T.tsv_blob(got.keys, got.counts, k) == O.tsv_blob(want)


@pytest.mark.parametrize("k,m", [(31, 21), (63, 21)])
@pytest.mark.parametrize("unit", [b"A", b"AC", b"ACGTT"])
def test_one_bin_of_many_instances(k, m, unit):
    """A microsatellite of half a million k-mer instances and a handful of distinct
    ones, between other sequence: one bin that many CTAs share."""
    import tuna_gb300 as T
    from tuna_gb300 import synth
    flank = synth.genome(40_000, 3, 0.5)
    sat = np.frombuffer(unit * (500_000 // len(unit)), dtype=np.uint8)
    seq = np.concatenate([flank[:20_000], sat, flank[20_000:]])
    with T.Context(0) as ctx:
        got, _ = ctx.run(k, m, seq=seq)
    want = O.count_stream(seq, k, m, threads=8)
    assert got.stats["heavy_groups"] >= 1 and got.stats["fallback_groups"] >= 1
    assert T.tsv_blob(got.keys, got.counts, k) == O.tsv_blob(want)


@pytest.mark.parametrize("k,m", [(31, 21), (41, 21)])
def test_group_sizes_at_the_store(k, m):
    """Streams whose k-mers fill one group to just below, at and above what a counting
    CTA's store holds (4096 one-word, 3072 two-word keys), all distinct and all twice."""
    import tuna_gb300 as T
    from tuna_gb300 import synth
    g = synth.genome(9_000, 11, 0.5)
    with T.Context(0) as ctx:
        for n in (1, 31, 32, 511, 512, 3071, 3072, 3073, 4095, 4096, 4097):
            for rep in (1, 2):
                s = np.tile(np.append(g[: n + k - 1], np.uint8(10)), rep)
                got, _ = ctx.run(k, m, seq=s, gpu_parts=1)
                want = O.count_stream(s, k, m, threads=2)
                assert T.tsv_blob(got.keys, got.counts, k) == O.tsv_blob(want), (n, rep)
