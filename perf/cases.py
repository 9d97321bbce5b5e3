"""The counting calls that users of this library make, over the sizes at which they make them.

Each case is one whole call of a public entry point on inputs of the workloads this repository
is measured on (the shapes of tuna_gb300/synth.py, drawn here on the GPU because they are made
many times): Illumina-like read sets, a repetitive assembly, requests of a counting service,
many small samples in one call. `kind` names the entry point:

  device    tg_count_seq_device_noalloc: a sequence stream and the pair buffers in device memory
  request   tg_count_seq: a sequence stream and the pair buffers in page-locked host memory
  fastq     tg_count_fastx: the bytes of a FASTQ file in page-locked host memory
  fasta     tg_count_fastx: the bytes of a FASTA file in page-locked host memory
  resident  Context.run on a stream in device memory; the pairs stay there, and the call's
            answer is the library's digest of them and the totals of the job
  batch     tg_count_batch: many samples in one call, pairs sample by sample
  tsv       Context.run with the text output (k-mer, tab, count) drained to host memory

The library returns pairs in any order, another one in each run. run() hands them over as they
come, as a user takes them; the dict that holds them gives them in the order of their k-mers when
they are read, and followed by zeros up to a size that the case alone gives, so that two runs can
be compared.
"""
import ctypes
import math

import numpy as np
import torch

import tuna_gb300 as T

U64_MAX = (1 << 64) - 1
DEV = "cuda:0"


# ---------------------------------------------------------------- cases

def listed():
    return [
        # a plugin or another library counts a contig or a few reads that it holds on the device:
        # the smallest calls, and the longest that the entry point takes
        dict(name="device_16k_k31", kind="device", bases=16_111, k=31, m=21, ci=1),
        dict(name="device_500k_k63", kind="device", bases=500_003, k=63, m=21, ci=1),
        # the counting service: reads of 100-250 bp; sizes around its median of 20 Mbp and the
        # three (k, m) that its requests name
        dict(name="request_1.5m_k25", kind="request", bases=1_500_007, k=25, m=21, ci=1),
        dict(name="request_20m_k31", kind="request", bases=20_000_003, k=31, m=21, ci=1),
        dict(name="request_150m_k21", kind="request", bases=150_000_001, k=21, m=17, ci=1),
        # a (k, m) without a cut kernel of its own, two-word keys
        dict(name="request_40m_k47_m31", kind="request", bases=40_000_037, k=47, m=31, ci=1),
        # the small read set: 4.6 Mbp genome at 30x, one FASTQ file
        dict(name="fastq_138m_k31", kind="fastq", bases=138_000_000, k=31, m=21, ci=1),
        # the large-k read set at a tenth of its size, k-mers seen once left out
        dict(name="fastq_300m_k63_ci2", kind="fastq", bases=300_000_000, k=63, m=21, ci=2),
        # the repetitive assembly at a tenth of its size, one FASTA file
        dict(name="fasta_310m_k31_m23", kind="fasta", bases=310_000_000, k=31, m=23, ci=1),
        # the whole 3.1 Gbp assembly on the device: the headline workload
        dict(name="resident_3100m_k31_m23", kind="resident", bases=3_100_000_000, k=31, m=23, ci=1),
        # the mix of independent samples, 1-200 kbp genomes at 5-50x
        dict(name="batch_400_k31", kind="batch", samples=400, k=31, m=21, ci=1),
        # text output of a read set, k-mers seen once left out
        dict(name="tsv_9m_k31_ci2", kind="tsv", bases=9_000_011, k=31, m=21, ci=2),
    ]


KM_SERVED = [(21, 17), (25, 21), (31, 21)]
KM_OTHER = [(31, 23), (33, 21), (47, 31), (63, 21), (15, 9), (27, 15)]


def _log(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng):
    kind = rng.choice(["device", "device", "request", "request", "fastq", "fasta", "resident", "batch", "tsv"])
    k, m = rng.choice(KM_SERVED if rng.random() < 0.6 else KM_OTHER)
    c = dict(kind=kind, k=k, m=m, ci=rng.choice([1, 1, 2]))
    if kind == "batch":
        c.update(samples=_log(rng, 20, 400), ci=1)
    elif kind == "device":
        c.update(bases=_log(rng, 1_000, 520_000))
    elif kind == "request":
        c.update(bases=_log(rng, 200_000, 150_000_000))
    elif kind == "fastq":
        c.update(bases=_log(rng, 2_000_000, 138_000_000) // 150 * 150)
    elif kind == "fasta":
        c.update(bases=_log(rng, 5_000_000, 310_000_000))
    elif kind == "resident":
        c.update(bases=_log(rng, 30_000_000, 2_000_000_000))
    else:
        c.update(bases=_log(rng, 1_000_000, 20_000_000), ci=2)
    return c


# ---------------------------------------------------------------- inputs

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _lut(text):
    return torch.tensor(list(text), dtype=torch.uint8, device=DEV)


def _random_bases(n, g, gc=0.5):
    """n i.i.d. ASCII bases with a share `gc` of G and C."""
    at = int(round((1 - gc) * 128))
    table = _lut(b"A" * at + b"T" * at + b"G" * (128 - at) + b"C" * (128 - at))
    return table[torch.randint(0, 256, (n,), generator=g, device=DEV, dtype=torch.uint8).int()]


CELL, FAM_A, FAM_B, B_CELLS = 300, 200, 40, 20


def _assembly(n, seed):
    """ASCII genome, GC 41 %: a quarter of it copies of 200 families of 300 bp, a fifth copies of 40
    families of 6 kbp, at 10-20 % divergence, 3 % microsatellites of 1-6 bp units."""
    g = _gen(seed)
    lib = torch.cat([_random_bases(FAM_A * CELL, g, 0.41), _random_bases(FAM_B * B_CELLS * CELL, g, 0.41)])
    out = torch.empty(n, dtype=torch.uint8, device=DEV)
    sup = B_CELLS * CELL                       # one superblock: a 6 kbp copy, or 20 cells
    step = max(1, (1 << 26) // sup)
    offs = torch.arange(CELL, device=DEV)
    for s0 in range(0, (n + sup - 1) // sup, step):
        ns = min(step, (n + sup - 1) // sup - s0)
        nc = ns * B_CELLS
        u = torch.rand(ns, generator=g, device=DEV)
        fam_b = torch.randint(0, FAM_B, (ns,), generator=g, device=DEV)
        src_b = FAM_A * CELL + (fam_b[:, None] * B_CELLS + torch.arange(B_CELLS, device=DEV)[None]) * CELL
        v = torch.rand(nc, generator=g, device=DEV)
        src_a = torch.randint(0, FAM_A, (nc,), generator=g, device=DEV) * CELL
        is_b = (u < 0.20)[:, None].expand(ns, B_CELLS).reshape(-1)
        is_a = ~is_b & (v < 0.3125)            # a quarter of all cells
        micro = ~is_b & (v > 0.9625)           # 3 % of all cells
        src = torch.where(is_b, src_b.reshape(-1), src_a)
        div = 0.10 + 0.10 * torch.rand(nc, generator=g, device=DEV)
        fresh = _random_bases(nc * CELL, g, 0.41).view(nc, CELL)
        keep = torch.rand((nc, CELL), generator=g, device=DEV) >= div[:, None]
        copied = lib[src[:, None] + offs[None]]
        cell = torch.where((is_a | is_b)[:, None] & keep, copied, fresh)
        unit = torch.randint(1, 7, (nc,), generator=g, device=DEV)
        rep = fresh.gather(1, offs[None] % unit[:, None])
        cell = torch.where(micro[:, None], rep, cell).reshape(-1)
        lo = s0 * sup
        hi = min(n, lo + cell.numel())
        out[lo:hi] = cell[: hi - lo]
    return out


def _contigs(n):
    """Lengths of 24 contigs, from 1 : 5 in size, that add up to n."""
    w = [1.0 + 4.0 * ((7 * i) % 24) / 23.0 for i in range(24)]
    lens = [int(n * x / sum(w)) for x in w]
    lens[-1] += n - sum(lens)
    return [x for x in lens if x > 0]


def _assembly_stream(n, seed):
    """The assembly as a sequence stream: contigs separated by line feeds."""
    a, parts, at = _assembly(n, seed), [], 0
    sep = _lut(b"\n")
    for ln in _contigs(n):
        parts += [a[at : at + ln], sep]
        at += ln
    return torch.cat(parts)


def _assembly_fasta(n, seed):
    """The assembly as the bytes of a FASTA file of 60 columns."""
    a, parts, at = _assembly(n, seed), [], 0
    for i, ln in enumerate(_contigs(n)):
        rows = ln // 60
        parts.append(_lut(b">contig_%d synthetic\n" % (i + 1)))
        body = torch.full((rows, 61), 10, dtype=torch.uint8, device=DEV)
        body[:, :60] = a[at : at + rows * 60].view(rows, 60)
        parts += [body.reshape(-1), a[at + rows * 60 : at + ln], _lut(b"\n")]
        at += ln
    return torch.cat(parts)


_COMP = None


def _reads(genome, starts, lens, err, n_rate, g):
    """A stream of reads: read i is genome[starts[i] : + lens[i]], from either strand, with
    substitutions at rate err[i] and N at n_rate, followed by a line feed."""
    global _COMP
    if _COMP is None:
        t = list(range(256))
        for a, b in zip(b"ACGT", b"TGCA"):
            t[a] = b
        _COMP = torch.tensor(t, dtype=torch.uint8, device=DEV)
    nr = lens.numel()
    ends = torch.cumsum(lens + 1, 0)
    read = torch.repeat_interleave(torch.arange(nr, device=DEV), lens + 1)
    pos = torch.arange(read.numel(), device=DEV) - (ends - lens - 1)[read]
    last = pos == lens[read]
    rev = (torch.rand(nr, generator=g, device=DEV) < 0.5)[read]
    at = starts[read] + torch.where(rev, lens[read] - 1 - pos, pos)
    b = genome[at.clamp_(0, genome.numel() - 1)]
    b = torch.where(rev, _COMP[b.int()], b)
    x = torch.rand(b.numel(), generator=g, device=DEV)
    b = torch.where(x < err[read], _random_bases(b.numel(), g), b)
    if n_rate:
        b = torch.where(x > 1 - n_rate, torch.full_like(b, ord("N")), b)
    b[last] = 10
    return b


def _read_stream(bases, seed, coverage, lo, hi, err, n_rate=0.0):
    """Reads of lo..hi bp at `coverage` over one random genome: about `bases` bases."""
    g = _gen(seed)
    glen = max(1000, bases // coverage)
    genome = _random_bases(glen, g)
    nr = max(1, int(bases / ((lo + hi) / 2)))
    lens = torch.randint(lo, hi + 1, (nr,), generator=g, device=DEV)
    starts = (torch.rand(nr, generator=g, device=DEV, dtype=torch.float64) * max(1, glen - hi)).long()
    return _reads(genome, starts, lens, torch.full((nr,), err, device=DEV), n_rate, g)


def _fastq(bases, seed):
    """FASTQ bytes of 150 bp reads at 30x, 0.5 % substitutions, 0.01 % N, Phred 30."""
    s = _read_stream(bases, seed, 30, 150, 150, 0.005, 0.0001).view(-1, 151)
    nr = s.shape[0]
    rows = torch.full((nr, 11 + 151 + 2 + 151), ord("?"), dtype=torch.uint8, device=DEV)
    rows[:, 0:2] = _lut(b"@r")
    i = torch.arange(nr, device=DEV)
    for d in range(8):
        rows[:, 9 - d] = (48 + (i // 10 ** d) % 10).to(torch.uint8)
    rows[:, 10] = 10
    rows[:, 11:162] = s
    rows[:, 162:164] = _lut(b"+\n")
    rows[:, -1] = 10
    return rows.reshape(-1)


def _sample_sizes(samples):
    """Genome length, reads and error rate of each sample: the same for every seed."""
    rng = np.random.default_rng(samples)
    glen = np.maximum(1000, np.exp(rng.uniform(math.log(40), math.log(200_000), samples)).astype(np.int64))
    cov, err = rng.uniform(5, 50, samples), rng.uniform(0.003, 0.01, samples)
    return glen, np.maximum(1, (glen * cov / 150).astype(np.int64)), err


def _batch(samples, seed):
    """Streams of independent samples: 150 bp reads of genomes of 1-200 kbp (log-uniform) at 5-50x
    with 0.3-1 % substitutions. Returns the joined stream and the samples' lengths."""
    g = _gen(seed)
    glen, nr, err = _sample_sizes(samples)
    genome = _random_bases(int(glen.sum()), g)
    off = torch.from_numpy(np.concatenate([[0], np.cumsum(glen)[:-1]])).to(DEV)
    s = torch.repeat_interleave(torch.arange(samples, device=DEV), torch.from_numpy(nr).to(DEV))
    room = torch.from_numpy(glen - 150).to(DEV)[s]
    starts = off[s] + (torch.rand(s.numel(), generator=g, device=DEV, dtype=torch.float64) * room).long()
    lens = torch.full((s.numel(),), 150, device=DEV)
    return _reads(genome, starts, lens, torch.from_numpy(err).float().to(DEV)[s], 0.0, g), nr * 151


# ---------------------------------------------------------------- calls

def _most_pairs(case):
    """More pairs than any inputs of the case give."""
    n = case.get("bases") or int((_sample_sizes(case["samples"])[1] * 150).sum())
    return n + n // 50 + 4096


def _padded(t, n):
    out = torch.zeros((n,) + t.shape[1:], dtype=t.dtype, device=t.device)
    out[: t.shape[0]] = t
    return out


class Pairs(dict):
    """The (k-mer, count) pairs of a call, with the job's totals. Reading "keys", "counts" or "text"
    gives them in the order of the k-mers (of each sample), then zeros."""

    def __init__(self, case, n, raw, **totals):
        super().__init__(n=n, **{k: None for k in raw}, **totals)
        self.raw, self.room = raw, _most_pairs(case)

    def __getitem__(self, name):
        if name == "text":  # the lines, sorted
            text = b"".join(sorted(self.raw["text"].splitlines(True)))
            return np.frombuffer(text.ljust(6 * self.room, b"\0"), dtype=np.uint8)
        if name not in ("keys", "counts"):
            return super().__getitem__(name)
        keys, counts = (x if isinstance(x, torch.Tensor) else torch.from_numpy(x).to(DEV)
                        for x in (self.raw["keys"], self.raw["counts"]))
        keys = keys.view(-1, keys.shape[-1])
        order = torch.arange(counts.numel(), device=DEV)
        for w in range(keys.shape[1]):
            order = order[torch.sort(keys[order, w], stable=True).indices]
        if "offsets" in self:
            off = torch.from_numpy(super().__getitem__("offsets")).to(DEV)
            sample = torch.repeat_interleave(torch.arange(off.numel() - 1, device=DEV), off[1:] - off[:-1])
            order = order[torch.sort(sample[order], stable=True).indices]
        return _padded((keys if name == "keys" else counts)[order], self.room)


_held = {}


def _host_room(nbytes):
    """Page-locked host memory for results, kept by the program from call to call."""
    if "room" not in _held or _held["room"].nbytes < nbytes:
        if "room" in _held:
            _held.pop("room").close()
        _held["room"] = T.HostBuffer(nbytes)
    return _held["room"]


def _to_host(t):
    """A GPU tensor's bytes in page-locked host memory."""
    hb = T.HostBuffer(t.numel())
    torch.from_numpy(hb.array()).copy_(t)
    return hb


def prepare(case, seed):
    kind, n = case["kind"], case.get("bases", 0)
    W = 1 if case["k"] <= 31 else 2
    s = dict(case=case, W=W, ctx=T.default_context(), L=T.library(), kind=kind,
             opts=T._JobOpts(case["k"], case["m"], 0, case["ci"], U64_MAX, 0, 0))
    if kind == "device":
        s["seq"] = _read_stream(n, seed, 20, 100, 250, 0.005)[:n].contiguous()
        s["keys"] = torch.zeros((n, W), dtype=torch.int64, device=DEV)
        s["counts"] = torch.zeros(n, dtype=torch.int32, device=DEV)
        s["err"] = ctypes.create_string_buffer(256)
        return s
    if kind == "resident":
        s["seq"] = _assembly_stream(n, seed)
        return s
    if kind == "batch":
        stream, lens = _batch(case["samples"], seed)
        s["in"] = _to_host(stream)
        at = s["in"].ptr + np.concatenate([[0], np.cumsum(lens)[:-1]]).astype(np.uint64)
        s["ptrs"] = (ctypes.c_void_p * len(lens))(*[int(p) for p in at])
        s["lens"] = (ctypes.c_size_t * len(lens))(*[int(x) for x in lens])
        s["offsets"] = np.zeros(len(lens) + 1, dtype=np.int64)
    elif kind in ("request", "tsv"):
        s["in"] = _to_host(_read_stream(n, seed, 20, 100, 250, 0.005))
    elif kind == "fastq":
        s["in"] = _to_host(_fastq(n, seed))
    else:
        s["in"] = _to_host(_assembly_fasta(n, seed))
    s["cap"] = (s["in"].nbytes + 255) // 256 * 256
    if kind != "tsv":
        _host_room(s["cap"] * (8 * W + 4))
    return s


def run(s):
    kind, L, ctx, W, case = s["kind"], s["L"], s["ctx"], s["W"], s["case"]
    n = ctypes.c_uint64()
    if kind == "device":
        rc = L.tg_count_seq_device_noalloc(ctypes.byref(s["opts"]), s["seq"].data_ptr(), s["seq"].numel(),
                                           s["keys"].data_ptr(), s["counts"].data_ptr(), s["counts"].numel(),
                                           ctypes.byref(n), torch.cuda.current_stream().cuda_stream, s["err"], 256)
        if rc:
            raise T.GpuError(rc, s["err"].value.decode())
        return Pairs(case, n.value, {"keys": s["keys"][: n.value], "counts": s["counts"][: n.value]})
    if kind == "resident":
        r, _ = ctx.run(case["k"], case["m"], dev_seq=s["seq"].data_ptr(), dev_len=s["seq"].numel(), n_parts=4096,
                       ci=case["ci"], want_results=False, digest=True)
        signed = [int(r.digest[h], 16) - (1 << 64) * (int(r.digest[h], 16) >> 63) for h in ("h1", "h2")]
        return dict(pairs=r.digest["pairs"], count_sum=r.digest["count_sum"], h1=signed[0], h2=signed[1],
                    kmers=r.stats["kmers"], records=r.stats["superkmers"], runs=r.stats["runs"],
                    bases=r.stats["bases"], distinct=r.stats["distinct"])
    if kind == "tsv":
        r, _ = ctx.run(case["k"], case["m"], seq=s["in"].array(), ci=case["ci"], want_results=False, drain=0)
        return Pairs(case, r.stats["out"], {"text": r.formatted}, kmers=r.stats["kmers"])
    room, cap, st = _host_room(0), s["cap"], T._Stats()
    keys, counts = room.ptr, room.ptr + cap * 8 * W
    if kind == "batch":
        rc = L.tg_count_batch(ctx.h, ctypes.byref(s["opts"]), len(s["lens"]), s["ptrs"], s["lens"], keys, counts,
                              s["offsets"].ctypes.data, cap, ctypes.byref(n), ctypes.byref(st))
    else:
        call = L.tg_count_seq if kind == "request" else L.tg_count_fastx
        rc = call(ctx.h, ctypes.byref(s["opts"]), s["in"].ptr, s["in"].nbytes, keys, counts, cap, ctypes.byref(n),
                  ctypes.byref(st))
    ctx.check(rc)
    raw = {"keys": room.array(np.int64, n.value * W).reshape(-1, W),
           "counts": room.array(np.uint8)[cap * 8 * W :].view(np.int32)[: n.value]}
    more = {"offsets": s["offsets"]} if kind == "batch" else {}
    return Pairs(case, n.value, raw, kmers=st.kmers, records=st.superkmers, distinct=st.distinct, **more)


# ---------------------------------------------------------------- work and exact results

def work(case):
    """The input read once and the pairs written once (8 or 16 + 4 bytes; k + 3 of text)."""
    k, kind = case["k"], case["kind"]
    n = case.get("bases") or float((_sample_sizes(case["samples"])[1] * 151).sum())
    pair = 12 if k <= 31 else 20
    if kind in ("fasta", "resident"):   # nearly every k-mer is new; a second copy of one is rare
        bytes_in, pairs = n * (61 / 60 if kind == "fasta" else 1), n * (0.95 if case["ci"] == 1 else 0.02)
    else:                               # the genome's k-mers, and k of them for every wrong base
        rate, cov, length = {"fastq": (0.005, 30, 150), "batch": (0.0065, 27.5, 150)}.get(kind, (0.005, 20, 175))
        seen = max(0.0, 1 - (k - 1) / length)
        pairs = n * (1 / cov + (0.75 * rate * k * seen * 0.9 if case["ci"] == 1 else 0.0))
        bytes_in = n * (315 / 150 if kind == "fastq" else 1)
    return {"bytes": float(bytes_in + pairs * (k + 3 if kind == "tsv" else pair)), "flops": 0.0}


def exact(case, seed):
    """The pairs by sorting all canonical k-mers, for streams of reads and k <= 31."""
    k, kind, n = case["k"], case["kind"], case.get("bases", 0)
    if kind not in ("device", "request") or k > 31 or n > 50_000_000:
        return None
    seq = _read_stream(n, seed, 20, 100, 250, 0.005)
    seq = (seq[:n] if kind == "device" else seq).long()
    code = torch.full((256,), -1, dtype=torch.int64, device=DEV)
    for i, c in enumerate(b"ACGT"):
        code[c] = (0, 1, 2, 3)[i]
    b = code[seq]
    bad = torch.cumsum(torch.cat([torch.zeros(1, dtype=torch.int64, device=DEV), (b < 0).long()]), 0)
    m = b.numel() - k + 1
    out = {"n": None, "keys": None, "counts": None}
    if m > 0:
        f, r = torch.zeros(m, dtype=torch.int64, device=DEV), torch.zeros(m, dtype=torch.int64, device=DEV)
        for i in range(k):
            x = b[i : i + m].clamp(min=0)
            f = f * 4 + x
            r = r + ((3 - x) << (2 * i))
        kept = torch.minimum(f, r)[bad[k:] == bad[:m]]
        keys, counts = torch.unique(kept, return_counts=True)
        keep = counts >= case["ci"]
        room = _most_pairs(case)
        out = {"n": int(keep.sum()), "keys": _padded(keys[keep][:, None], room),
               "counts": _padded(counts[keep].int(), room)}
    if kind == "request":
        out.update(kmers=None, records=None, distinct=None)
    return out
