// tg_phase2.cu — Phase 2 on the GPU: exact count of every canonical k-mer of
// every bucket record, ci/cx filter and compaction of the surviving pairs.
//
// Reference behaviour (paths relative to the reference project root):
//   every k-mer of a record       src/count.hpp:71-175 (rolled through the record's
//                                 packed bases, one record per thread)
//   canonical form                include/kache-hash/Kmer.hpp:446-456, :629-646
//                                 (min of k-mer and reverse complement, word order)
//   count += 1 per instance       src/count.hpp:81, Streaming_Kmer_Hash_Table::upsert
//   keep ci <= count <= cx        src/count.hpp:202, :250, :287
//
// Pipeline (all instances of a canonical k-mer share its minimizer, hence its
// bin: the sample's first bin + minimizer hash bits; phase 1 counted the k-mer
// instances of every bin):
//   k_scan*     bin counts -> k-mer and record offsets
//   k_plan      per segment (a run of bins of one sample): groups of whole bins
//               of at most `target` k-mers
//   k_recs      every record with its bases at its group's cursor, so the records
//               of a group are one contiguous range
//   k_count     persistent: each group's records are read with coalesced loads
//               and unpacked into canonical keys in shared memory, counted in an
//               open-addressing table there, then filtered and compacted.
//   k_rounds    larger groups (one bin), a CTA each: in rounds when their distinct
//               keys fit in the store, else as key-hash parts written to global
//               memory first or, without room for that, read again in the next
//               launch; past MAX_PARTS parts they go to the global table (k_fb_*)
//   k_big       the largest, each shared by many CTAs, into one global table
#include <algorithm>
#include <vector>

#include "tg_launch.h"

namespace tg {

constexpr int COUNT_THREADS = 512;       // threads of a k_count CTA
constexpr int COUNT_PER_SM = 2;          // CTAs per SM: one counts while the other waits at a barrier
constexpr uint32_t MAX_PARTS = 128;      // key-hash parts of one range before the global table
constexpr uint64_t FALLBACK_CAP = 4096;
constexpr uint32_t BIG_KEYS = 1u << 16;  // k-mers above which many CTAs share a group (k_big)
constexpr uint64_t WAVE_KEYS = 1u << 22; // k-mers of a wave of the first counting pass (P2Overlap)
constexpr uint32_t MAX_SPLIT = 32;       // parts that split_group makes of a group
constexpr uint64_t SPLIT_MIN = 1u << 20; // k-mers of a job that has room for that
// Packed records of such a group that a CTA takes at a time (counting 155 Mbp of the
// assembly, k=31 m=23: 1.61 ms against 1.92 with 4,096; 12.8 Mbp of reads, k=15 m=9:
// 0.63 ms, 0.72 with 1,024).
constexpr uint32_t BIG_CHUNK = 512;
// k-mers of such groups that share a table: larger tables leave L2 (100 Mbp, k=21 m=9,
// nearly all of whose k-mers are in such groups: 10.5 ms of counting, 11.8 with one table).
constexpr uint64_t BIG_TABLE_KEYS = 1u << 23;


struct __align__(16) U128 {
    unsigned long long lo, hi;
};

template <int W>
struct KeyOps;

template <>
struct KeyOps<1> {
    using Key = unsigned long long;
    static constexpr size_t BYTES = 8;
    __device__ static Key empty() { return ~0ull; }
    __device__ static bool is_empty(const Key& k) { return k == ~0ull; }
    __device__ static bool eq(const Key& a, const Key& b) { return a == b; }
    __device__ static uint64_t hash(const Key& k) { return mix_key1(k); }
    __device__ static Key load(const Key* p) { return *reinterpret_cast<const volatile Key*>(p); }
    __device__ static Key cas(Key* p, const Key& cmp, const Key& val) { return atomicCAS(p, cmp, val); }
    __device__ static void store(void* out, uint64_t i, const Key& k) {
        reinterpret_cast<unsigned long long*>(out)[i] = k;
    }
};

template <>
struct KeyOps<2> {
    using Key = U128;
    static constexpr size_t BYTES = 16;
    __device__ static Key empty() { Key k; k.lo = ~0ull; k.hi = ~0ull; return k; }
    __device__ static bool is_empty(const Key& k) { return k.hi == ~0ull; }
    __device__ static bool eq(const Key& a, const Key& b) { return a.lo == b.lo && a.hi == b.hi; }
    __device__ static uint64_t hash(const Key& k) { K2 x{k.lo, k.hi}; return mix_key2(x); }
    __device__ static Key load(const Key* p) {
        const volatile unsigned long long* q = reinterpret_cast<const volatile unsigned long long*>(p);
        Key k; k.lo = q[0]; k.hi = q[1]; return k;
    }
    __device__ static Key cas(Key* p, const Key& cmp, const Key& val) { return atomicCAS(p, cmp, val); }
    __device__ static void store(void* out, uint64_t i, const Key& k) {
        reinterpret_cast<U128*>(out)[i] = k;
    }
};

// Key-hash part of a key (hash bits apart from the table's slot bits).
template <int W>
__device__ __forceinline__ uint32_t key_part(const typename KeyOps<W>::Key& key, uint32_t parts) {
    return (uint32_t)(KeyOps<W>::hash(key) >> 8) & (parts - 1);
}

// Insert n instances of one k-mer: count += n. False if `limit` slots were taken. (A
// table of global memory takes its mask for that, one less than its slots, 2^32 of which
// have no number of 32 bits; more than half of them are free.)
// 64-bit keys are probed with a plain load and claimed with a CAS. A 128-bit
// key cannot be read in one single-copy-atomic load, and a read torn against a
// concurrent claim could skip the slot that holds the same k-mer, so 128-bit
// slots are probed with the CAS itself: it returns the whole current key.
template <int W>
__device__ __forceinline__ bool tbl_add(typename KeyOps<W>::Key* keys, uint32_t* cnt, uint32_t mask,
                                        const typename KeyOps<W>::Key& key, uint32_t n, uint32_t limit) {
    using O = KeyOps<W>;
    uint32_t h = (uint32_t)(O::hash(key) >> 32) & mask;
    for (uint32_t p = 0; p < limit; ++p) {
        if constexpr (W == 1) {
            const typename O::Key cur = O::load(&keys[h]);
            if (O::eq(cur, key)) { atomicAdd(&cnt[h], n); return true; }
            if (O::is_empty(cur)) {
                const typename O::Key prev = O::cas(&keys[h], O::empty(), key);
                if (O::is_empty(prev) || O::eq(prev, key)) { atomicAdd(&cnt[h], n); return true; }
            }
        } else {
            const typename O::Key prev = O::cas(&keys[h], O::empty(), key);
            if (O::is_empty(prev) || O::eq(prev, key)) { atomicAdd(&cnt[h], n); return true; }
        }
        h = (h + 1) & mask;
    }
    return false;
}

// ---------------------------------------------------------------- packed records
template <int W>
struct Rec {
    unsigned long long w[2 * W];
    __device__ __forceinline__ uint32_t n() const { return (uint32_t)w[2 * W - 1] & 63u; }
};
template <int W>
__device__ __forceinline__ Rec<W> load_rec(const void* recs, unsigned long long i) {
    const ulonglong2* p = static_cast<const ulonglong2*>(recs) + i * W;
    Rec<W> r;
#pragma unroll
    for (int j = 0; j < W; ++j) {
        const ulonglong2 v = __ldg(p + j);
        r.w[2 * j] = v.x;
        r.w[2 * j + 1] = v.y;
    }
    return r;
}

// The k-mers of a packed record one after the other: the k-mer, its reverse
// complement and the bases still to come (at most REC_MAX - 1), shifted by one
// base per step.
template <int W>
struct Roll;

template <>
struct Roll<1> {
    uint32_t f0, f1;  // the k-mer, low word first
    uint32_t r0, r1;  // its reverse complement, left-aligned
    uint32_t x;       // the bases to come, left-aligned
    __device__ __forceinline__ void start(const Rec<1>& c, int k) {
        const unsigned long long f = c.w[0] >> (64 - 2 * k), r = revcomp64(f, k) << (64 - 2 * k);
        f0 = (uint32_t)f;
        f1 = (uint32_t)(f >> 32);
        r0 = (uint32_t)r;
        r1 = (uint32_t)(r >> 32);
        x = (uint32_t)(((c.w[0] << (2 * k)) | (c.w[1] >> (64 - 2 * k))) >> 32);
    }
    __device__ __forceinline__ unsigned long long key(int k) const {
        const unsigned long long f = ((unsigned long long)f1 << 32) | f0;
        const unsigned long long r = (((unsigned long long)r1 << 32) | r0) >> (64 - 2 * k);
        return f < r ? f : r;
    }
    __device__ __forceinline__ void step(int k) {
        const unsigned long long mask = ~0ull >> (64 - 2 * k);
        f1 = __funnelshift_l(f0, f1, 2) & (uint32_t)(mask >> 32);
        f0 = __funnelshift_l(x, f0, 2) & (uint32_t)mask;
        r0 = __funnelshift_r(r0, r1, 2);
        r1 = (r1 >> 2) | (~x & 0xC0000000u);
        x <<= 2;
    }
};

template <>
struct Roll<2> {
    K2 f, r;
    uint32_t x;
    __device__ __forceinline__ void start(const Rec<2>& c, int k) {
        const int sh = 128 - 2 * k;  // 2..64
        if (sh >= 64) { f.lo = c.w[0]; f.hi = 0; }
        else { f.lo = (c.w[1] >> sh) | (c.w[0] << (64 - sh)); f.hi = c.w[0] >> sh; }
        r = revcomp128(f, k);
        const int s = 2 * k - 64;    // 0..62
        x = (uint32_t)((s ? (c.w[1] << s) | (c.w[2] >> (64 - s)) : c.w[1]) >> 32);
    }
    __device__ __forceinline__ U128 key(int) const {
        const bool l = k2_less(f, r);
        U128 q;
        q.lo = l ? f.lo : r.lo;
        q.hi = l ? f.hi : r.hi;
        return q;
    }
    __device__ __forceinline__ void step(int k) {
        const uint32_t b = x >> 30;
        x <<= 2;
        f.hi = (f.hi << 2) | (f.lo >> 62);
        if (2 * k > 64) f.hi &= ~0ull >> (128 - 2 * k);
        else f.hi = 0;
        f.lo = (f.lo << 2) | b;
        r.lo = (r.lo >> 2) | (r.hi << 62);
        r.hi >>= 2;
        if (k == 32) r.lo |= (unsigned long long)(3u - b) << 62;
        else r.hi |= (unsigned long long)(3u - b) << (2 * k - 66);
    }
};

__device__ __forceinline__ uint32_t rec_hash(const Rec<1>& r) {
    return (uint32_t)r.w[0] * 0x9E3779B1u + (uint32_t)(r.w[0] >> 32) * 0x85EBCA77u +
           ((uint32_t)r.w[1] + (uint32_t)(r.w[1] >> 32)) * 0xC2B2AE3Du;
}
__device__ __forceinline__ uint32_t rec_hash(const Rec<2>& r) {
    return (uint32_t)r.w[0] * 0x9E3779B1u + (uint32_t)(r.w[0] >> 32) * 0x85EBCA77u + (uint32_t)r.w[1] * 0xC2B2AE3Du +
           (uint32_t)(r.w[1] >> 32) * 0x27D4EB2Fu + ((uint32_t)r.w[2] ^ (uint32_t)r.w[3]) * 0x165667B1u +
           (uint32_t)(r.w[2] >> 32) * 0x9E3779B1u;
}
template <int W>
__device__ __forceinline__ bool rec_equal(const Rec<W>& a, const Rec<W>& b) {
    bool e = true;
#pragma unroll
    for (int j = 0; j < 2 * W; ++j) e = e && a.w[j] == b.w[j];
    return e;
}

// ---------------------------------------------------------------- k_plan
// plan_split warps per segment (a run of consecutive bins of one sample), each
// with an equal share of its bins: the share's groups,
// from the scanned k-mer offsets ko[bin]. Greedy, in bin order: a group starting
// at bin s takes the most bins e - s with at most `target` k-mers (one bin if that
// bin alone is larger; a group that a CTA's store cannot hold is listed apart). Each step is one
// upper-bound search over ko, done by the warp as a 32-way search. Every bin of
// the group gets the group's first bin in gfirst: k_recs appends all of the
// group's records at that bin's cursor.
constexpr int PLAN_THREADS = 256;

__global__ void __launch_bounds__(PLAN_THREADS) k_plan(KeysParams P) {
    const int lane = threadIdx.x & 31;
    const uint32_t wi = blockIdx.x * (PLAN_THREADS / 32) + (threadIdx.x >> 5);
    const uint32_t sg = wi / P.plan_split, part = wi % P.plan_split;
    if (sg >= P.n_segs) return;  // warp-uniform
    Segment seg = P.segs[sg];
    {
        const uint32_t per = (seg.bin_hi - seg.bin_lo + P.plan_split - 1) / P.plan_split;
        const uint32_t hi = seg.bin_hi;
        seg.bin_lo = min(hi, seg.bin_lo + part * per);
        seg.bin_hi = min(hi, seg.bin_lo + per);
        if (seg.bin_lo == seg.bin_hi) return;
    }
    const uint32_t nb = seg.bin_hi - seg.bin_lo;
    const unsigned long long* ko = P.kofs + seg.bin_lo;
    const unsigned long long end = ko[nb];
    const unsigned long long T = P.target;
    uint32_t s = 0;
    unsigned long long ks = ko[0];
    while (ks < end) {
        // largest e in [s + 1, nb] with ko[e] <= ks + T (e = s + 1 if there is none)
        const unsigned long long lim = ks + T;
        uint32_t lo = s + 1, hi = nb;
        if (ko[lo] <= lim) {
            while (lo < hi) {  // invariant: ko[lo] <= lim, the answer is in [lo, hi]
                const uint32_t step = (hi - lo + 31) / 32;
                const uint32_t e = lo + (uint32_t)lane * step;
                const unsigned ok = __ballot_sync(0xffffffffu, e <= hi && ko[e] <= lim);  // bit 0 is set
                const int l = 31 - __clz(ok);
                const uint32_t nlo = lo + (uint32_t)l * step;
                hi = l == 31 ? hi : min(nlo + step - 1, hi);
                lo = nlo;
            }
        }
        const uint32_t e = lo;
        const unsigned long long ke = ko[e];
        for (uint32_t b = s + (uint32_t)lane; b < e; b += 32) P.gfirst[seg.bin_lo + b] = seg.bin_lo + s;
        if (lane == 0 && ke > ks) {  // not the empty bins before a bin larger than the target
            const int heavy = ke - ks > P.store ? (ke - ks > BIG_KEYS ? 2 : 1) : 0;
            const unsigned long long q = atomicAdd(&P.ctr[heavy == 2 ? P2C_BIG : heavy ? P2C_HEAVY : P2C_NORMAL], 1ull);
            if (q < P.groups_cap) {
                Group g;
                g.lo = P.rofs[seg.bin_lo + s];
                g.hi = P.rofs[seg.bin_lo + e];
                g.parts = 1;
                g.part = 0;
                g.sample = seg.sample;
                g.keys = (uint32_t)(ke - ks);
                P.groups[heavy][q] = g;
            }
        }
        s = e;
        ks = ke;
    }
}

// ---------------------------------------------------------------- k_recs
// Every record of the phase-1 descriptor lists (in stream order, so the packed
// bases are read front to back) as packed records at its group's cursor (the
// cursor of the group's first bin, gfirst), one thread per descriptor: the place
// from one global atomic, the bases from an unaligned window of the packed
// words. Four descriptors per thread in flight; the loads of a descriptor, its
// group, its place and its bases depend on one another and nothing else bounds
// the kernel but the scattered 16-byte writes.
constexpr int RECS_THREADS = 256, RECS_UNROLL = 4, RECS_PER_CTA = 2 * RECS_UNROLL * RECS_THREADS;

// The packed record of the nk k-mers from stream position s on.
template <int W>
__device__ __forceinline__ void store_rec(const KeysParams& P, unsigned long long at, uint64_t s, uint32_t nk) {
    const int bits = 2 * (P.k + (int)nk - 1);
    const uint64_t a = s + TG_PAD;
    const uint32_t* p = P.packed + (a >> 4);
    const uint32_t sh = 2 * (uint32_t)(a & 15);
    uint32_t x[4 * W + 1], y[4 * W];
#pragma unroll
    for (int i = 0; i <= 4 * W; ++i) x[i] = __ldg(p + i);
#pragma unroll
    for (int i = 0; i < 4 * W; ++i) {  // the record's bases alone: equal records are equal words
        y[i] = __funnelshift_l(x[i + 1], x[i], sh);
        const int v = bits - 32 * i;
        if (v < 32) y[i] &= v > 0 ? ~(0xFFFFFFFFu >> v) : 0u;
    }
    y[4 * W - 1] |= nk;
    ulonglong2* d = static_cast<ulonglong2*>(P.recs) + at * W;
#pragma unroll
    for (int j = 0; j < W; ++j)
        d[j] = make_ulonglong2(((unsigned long long)y[4 * j] << 32) | y[4 * j + 1],
                               ((unsigned long long)y[4 * j + 2] << 32) | y[4 * j + 3]);
}

template <int W>
__global__ void __launch_bounds__(RECS_THREADS) k_recs(KeysParams P) {
    const uint32_t n = P.n_desc ? (uint32_t)min((uint64_t)P.n_desc[blockIdx.y], P.desc_cap) : P.n_one;
    const uint64_t* d = P.desc + (uint64_t)blockIdx.y * P.desc_cap;
    const int sb = P.desc_sb;
    const uint64_t i0 = (uint64_t)blockIdx.x * RECS_PER_CTA;
#pragma unroll
    for (int b = 0; b < RECS_PER_CTA; b += RECS_UNROLL * RECS_THREADS) {
        if (i0 + b >= n) return;
        uint64_t dv[RECS_UNROLL];
        uint32_t g[RECS_UNROLL];
        unsigned long long at[RECS_UNROLL];
#pragma unroll
        for (int u = 0; u < RECS_UNROLL; ++u) {
            const uint64_t i = i0 + b + u * RECS_THREADS + threadIdx.x;
            dv[u] = i < n ? __ldcs(d + i) : 0;
            const uint32_t bin = desc_bin(dv[u], sb);
            if (bin < P.bin_lo || bin >= P.bin_hi) dv[u] = 0;  // not this run's: no k-mers
        }
#pragma unroll
        for (int u = 0; u < RECS_UNROLL; ++u)
            if (desc_nk(dv[u], sb)) g[u] = P.gfirst[desc_bin(dv[u], sb)];
#pragma unroll
        for (int u = 0; u < RECS_UNROLL; ++u) {
            const uint32_t nk = desc_nk(dv[u], sb);
            if (nk) at[u] = atomicAdd(&P.rofs[g[u]], (unsigned long long)rec_pieces(nk));
        }
#pragma unroll
        for (int u = 0; u < RECS_UNROLL; ++u) {
            const uint32_t nk = desc_nk(dv[u], sb);
            const uint64_t s = desc_start(dv[u], sb);
            if (!nk) continue;
            if (nk <= REC_MAX) {
                store_rec<W>(P, at[u], s, nk);
                continue;
            }
            const uint32_t pieces = rec_pieces(nk), per = (nk + pieces - 1) / pieces;
            for (uint32_t q = 0; q < pieces; ++q) {
                const uint32_t o = min(q * per, nk);
                store_rec<W>(P, at[u] + q, s + o, min(per, nk - o));
            }
        }
    }
}

// ---------------------------------------------------------------- k_count
__device__ __forceinline__ uint32_t smem_addr(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

// End of the launch's slice of the list.
__device__ __forceinline__ unsigned long long list_end(const CountParams& P) {
    return P.n_list ? min(P.g_end, *P.n_list) : P.g_end;
}

// Asynchronous copy (cp.async, two 16-byte pieces) of group `gi` of the launch's
// list into shared memory; an index past the end gives an empty group.
__device__ __forceinline__ void copy_group(Group* dst, const CountParams& P, unsigned long long gi,
                                           unsigned long long g_end) {
    if (gi >= g_end) {
        dst->lo = dst->hi = 0;
        return;
    }
    const Group* src = P.list + gi;
    const uint32_t d = smem_addr(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + 16),
                 "l"(reinterpret_cast<const uint8_t*>(src) + 16)
                 : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
}

// Shape of the counting kernel for key width W. The table holds 32-bit entries,
// not keys: an entry is the key's place in the CTA's key store (IDX_BITS) and a
// fingerprint of the key (the rest); the store holds each key once, at that
// place, with its count in a second array. So an insert is one 4-byte shared
// CAS at a random slot, a full key is read at random only where the fingerprint
// says that it is the same key, and the output walk reads keys and counts in
// order. CAP keys fit in the store, COUNT_PER_SM CTAs in an SM's shared memory;
// the table is at most a quarter (W = 1) or three eighths full, so that a warp's
// longest probe stays short.
template <int W>
struct CountShape;
template <>
struct CountShape<1> {
    static constexpr uint32_t SLOT_BITS = 14, CAP = 4096;
};
template <>
struct CountShape<2> {
    static constexpr uint32_t SLOT_BITS = 13, CAP = 3072;
};
constexpr int IDX_BITS = 13;                          // place in the key store
constexpr uint32_t IDX_MASK = (1u << IDX_BITS) - 1;
constexpr uint32_t DEDUP_MAX = 3;                     // records per thread among which equal ones are looked for
constexpr uint32_t NO_ENTRY = 0xFFFFFFFFu;            // an empty slot; no entry has all bits set (CAP <= IDX_MASK)

template <int W>
struct CountSmem {
    using Key = typename KeyOps<W>::Key;
    static constexpr uint32_t SLOTS = 1u << CountShape<W>::SLOT_BITS, CAP = CountShape<W>::CAP;
    Key keys[CAP];
    uint32_t table[SLOTS];
    uint32_t cnt[CAP];          // occurrences after the first
    Group grp[3];               // groups g, g + 1, g + 2
    unsigned long long pending;
    uint32_t staged;
    uint32_t part_end[MAX_SPLIT];  // split_group: keys, cursors, then ends of the parts
    uint32_t dedup, firsts;     // groups until equal records are looked for again; first ones found
    static_assert(CAP <= IDX_MASK && CAP < SLOTS, "places and free slots");
};

// Home slot and entry of a key at place i: both the top bits of a multiply-add
// hash. They share bits, so one in 32 keys that meet at a home slot are compared in
// full without being equal; a second mixing step costs more than that. The odd
// multipliers here and in rec_hash are xxHash's 32-bit primes (well-mixed constants;
// nothing else of it is used, and no result depends on them).
__device__ __forceinline__ uint32_t slot_hash(unsigned long long k) {
    return (uint32_t)k * 0x9E3779B1u + (uint32_t)(k >> 32) * 0x85EBCA77u;
}
__device__ __forceinline__ uint32_t slot_hash(const U128& k) {
    return slot_hash(k.lo) + (uint32_t)k.hi * 0xC2B2AE3Du + (uint32_t)(k.hi >> 32) * 0x27D4EB2Fu;
}
template <int W>
__device__ __forceinline__ void place_of(uint32_t x, uint32_t i, uint32_t& h, uint32_t& entry) {
    h = x >> (32 - CountShape<W>::SLOT_BITS);
    entry = (x & ~IDX_MASK) | i;
}

// The slot probed after h for the key of `entry`: the stride is odd, so the
// probe comes past every slot, and there are more slots than places, so it finds
// a free one.
template <int W>
__device__ __forceinline__ uint32_t next_slot(uint32_t h, uint32_t entry) {
    return (h + ((entry >> IDX_BITS) | 1u)) & (CountSmem<W>::SLOTS - 1);
}

template <int W>
__device__ __forceinline__ void clear_table(CountSmem<W>& S) {
    uint4* t4 = reinterpret_cast<uint4*>(S.table);
#pragma unroll 4
    for (uint32_t i = threadIdx.x; i < CountSmem<W>::SLOTS / 4; i += COUNT_THREADS)
        t4[i] = make_uint4(NO_ENTRY, NO_ENTRY, NO_ENTRY, NO_ENTRY);
}

template <int W>
__device__ __forceinline__ void start_store(CountSmem<W>& S) {
    clear_table<W>(S);
    for (uint32_t i = threadIdx.x; i < CountShape<W>::CAP; i += COUNT_THREADS) S.cnt[i] = 0;
    if (threadIdx.x == 0) S.staged = S.dedup = S.firsts = 0;
}

// Writes the new keys of the first n places (bit u of newm: this thread's place
// u * COUNT_THREADS + threadIdx.x holds one) that pass ci/cx to out, each warp's
// next to each other, and empties the table and the counts. All threads call it
// with the inserts done but for a barrier; after it, one barrier more and the
// store may be filled again. Every warp reserves its own place in out, before the
// barrier where it can, so that the atomic's round trip overlaps the wait there
// (one atomic per CTA, between two barriers more, cost 0.2 of 1.3 ms for 0.15 G
// distinct keys). behind() runs on every thread behind the barrier.
template <int W, typename F>
__device__ __forceinline__ void write_out(const CountParams& P, CountSmem<W>& S, uint32_t n, uint32_t newm,
                                          uint32_t sample, uint32_t& distinct, F&& behind) {
    using Key = typename KeyOps<W>::Key;
    constexpr uint32_t UMAX = CountShape<W>::CAP / COUNT_THREADS;
    const uint32_t tid = threadIdx.x, lane = tid & 31;
    const bool filtered = P.ci > 1 || P.cx < 0xFFFFFFFFull;  // counts are at least 1 and fit in 32 bits
    uint32_t wn = __reduce_add_sync(0xffffffffu, __popc(newm));
    unsigned long long wb = 0;
    distinct += wn;
    if (!filtered && lane == 0 && wn) wb = atomicAdd(&P.ctr[P2C_OUT], (unsigned long long)wn);
    __syncthreads();  // inserts done
    behind();
    clear_table<W>(S);
    if (filtered) {
        uint32_t keep = 0;
        for (uint32_t u = 0; u < UMAX; ++u)
            if ((newm >> u) & 1u) {
                const uint32_t i = u * COUNT_THREADS + tid;
                const uint64_t c = (uint64_t)S.cnt[i] + 1;
                if (c >= P.ci && c <= P.cx) keep |= 1u << u;
                else S.cnt[i] = 0;
            }
        newm = keep;
        wn = __reduce_add_sync(0xffffffffu, __popc(newm));
        if (lane == 0 && wn) wb = atomicAdd(&P.ctr[P2C_OUT], (unsigned long long)wn);
    }
    if (wn == 0) return;  // the whole warp
    if (P.sample_tot && lane == 0) atomicAdd(&P.sample_tot[sample], wn);
    wb = __shfl_sync(0xffffffffu, wb, 0);
    // every pair of the warp has room (the same for its lanes), or each is checked
    const uint32_t room = wb + wn <= P.out_cap ? ~0u : (uint32_t)(wb < P.out_cap ? P.out_cap - wb : 0);
    Key* okeys = static_cast<Key*>(P.out_keys) + wb;
    uint32_t* ocnt = P.out_counts + wb;
    uint32_t* osmp = P.out_sample ? P.out_sample + wb : nullptr;
    uint32_t before = 0;
    for (uint32_t u = 0; u * COUNT_THREADS < n; ++u) {
        const uint32_t i = u * COUNT_THREADS + tid;
        const bool kept = (newm >> u) & 1u;
        const unsigned bal = __ballot_sync(0xffffffffu, kept);
        const uint32_t o = before + __popc(bal & ((1u << lane) - 1));
        before += __popc(bal);
        if (kept) {
            const uint32_t c = S.cnt[i];
            if (o < room) {
                okeys[o] = S.keys[i];
                ocnt[o] = c + 1;
                if (osmp) osmp[o] = sample;
            }
            if (c) S.cnt[i] = 0;
        }
    }
}

// Persistent: COUNT_PER_SM CTAs per SM take groups of at most CAP k-mers from a global
// counter. A group's packed records are unpacked into the key store, a barrier, every
// thread inserts the keys at places t, t + COUNT_THREADS, ... and notes which of them
// are new, a barrier, and the new ones are written to out. The barrier between
// unpacking and inserting makes every stored key readable, so a fingerprint match can
// be checked against the store at once. Group entries are fetched two groups ahead
// (cp.async) into a ring of three, a group's first records while the one before is
// inserted.
//
// At most 56 registers per thread: 1,024 threads x 56 leave 8,192 of the SM's
// registers, room for one CTA of the host-link copy (tg_link.cu: 256 threads x 32
// registers) beside the counting CTAs, so the copy of a wave's pairs to host memory
// runs while the next wave counts.
template <int W>
__global__ void __maxnreg__(56) k_count(const __grid_constant__ CountParams P) {
    using O = KeyOps<W>;
    using Key = typename O::Key;
    constexpr uint32_t CAP = CountShape<W>::CAP, SLOTS = CountSmem<W>::SLOTS;
    constexpr uint32_t UMAX = CAP / COUNT_THREADS;           // places per thread
    constexpr int U = 2;                                     // of them in flight
    static_assert(CAP % (U * COUNT_THREADS) == 0 && UMAX <= 32, "one bit per place of a thread");
    extern __shared__ __align__(128) uint8_t smem[];
    CountSmem<W>& S = *reinterpret_cast<CountSmem<W>*>(smem);
    const int k = P.k;
    const uint32_t tid = threadIdx.x, lane = tid & 31;
    uint32_t distinct = 0;                                   // per warp

    const unsigned long long g_end = list_end(P);
    if (P.g_begin + blockIdx.x >= g_end) return;  // fewer groups than CTAs
    start_store<W>(S);
    if (tid == 0) {
        for (int q = 0; q < 3; ++q) copy_group(&S.grp[q], P, P.g_begin + atomicAdd(P.work, 1ull), g_end);
        S.pending = P.g_begin + atomicAdd(P.work, 1ull);     // index of group g + 3
        asm volatile("cp.async.wait_all;" ::: "memory");
    }
    __syncthreads();

    // this thread's first packed record of a group (no k-mers past the group's end)
    auto load_at = [&](const Group& g, uint32_t i) {
        Rec<W> c;
        c.w[2 * W - 1] = 0;
        if (i < (uint32_t)(g.hi - g.lo)) c = load_rec<W>(P.recs, g.lo + i);
        return c;
    };
    Rec<W> ahead = load_at(S.grp[0], tid);
    for (uint32_t q = 0;; q = q == 2 ? 0 : q + 1) {
        const Group& g = S.grp[q];
        if (g.hi == g.lo) break;  // no more groups
        const uint32_t sample = g.sample, nrec = (uint32_t)(g.hi - g.lo);
        // Equal records first, where the last groups had enough of them (read sets: a
        // record inside several reads): one of them is unpacked, with their number as the
        // weight of its keys. The table holds record numbers meanwhile, cnt their
        // occurrences after the first; both are empty again before the keys come.
        constexpr uint32_t DM = W == 1 ? DEDUP_MAX : 1;
        Rec<W> mine[DM];
        uint32_t weight[DM];
        const bool dedup = W == 1 && S.dedup == 0 && nrec <= DM * COUNT_THREADS;
        if (W == 1 && dedup) {
            Rec<W>* recs = reinterpret_cast<Rec<W>*>(S.keys);
            uint32_t first = 0;  // bit j: this thread's j-th record is the first of its kind
            mine[0] = ahead;
#pragma unroll
            for (uint32_t j = 1; j < DM; ++j) mine[j] = load_at(g, j * COUNT_THREADS + tid);
#pragma unroll
            for (uint32_t j = 0; j < DM; ++j)
                if (j * COUNT_THREADS + tid < nrec) recs[j * COUNT_THREADS + tid] = mine[j];
            __syncthreads();
#pragma unroll
            for (uint32_t j = 0; j < DM; ++j) {
                const uint32_t i = j * COUNT_THREADS + tid;
                weight[j] = 0;
                if (i >= nrec) continue;
                uint32_t h, en;
                place_of<W>(rec_hash(mine[j]), i, h, en);
                for (uint32_t p = 0; p < SLOTS; ++p) {
                    const uint32_t e = atomicCAS(&S.table[h], NO_ENTRY, en);
                    if (e == NO_ENTRY) {
                        weight[j] = 1;
                        ++first;
                        break;
                    }
                    if (((e ^ en) >> IDX_BITS) == 0 && rec_equal(recs[e & IDX_MASK], mine[j])) {
                        atomicAdd(&S.cnt[e & IDX_MASK], 1u);
                        break;
                    }
                    h = next_slot<W>(h, en);
                }
            }
            __syncwarp();
            first = __reduce_add_sync(0xffffffffu, first);
            if (lane == 0) atomicAdd(&S.firsts, first);
            __syncthreads();
#pragma unroll
            for (uint32_t j = 0; j < DM; ++j)
                if (weight[j]) {
                    weight[j] += S.cnt[j * COUNT_THREADS + tid];
                    S.cnt[j * COUNT_THREADS + tid] = 0;
                }
            clear_table<W>(S);
            if (tid == 0) {  // too few were equal: the next 15 groups without
                if (S.firsts > nrec - nrec / 4) S.dedup = 15;
                S.firsts = 0;
            }
            __syncthreads();
        }
        // A warp unpacks 32 records, each lane its own: the keys of a record one after
        // the other in the store, the warp's records next to each other.
        auto unpack = [&](const Rec<W>& rec, uint32_t nk, uint32_t w) {
            uint32_t x = nk;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            uint32_t at = 0;
            if (lane == 31) at = atomicAdd(&S.staged, x);
            at = __shfl_sync(0xffffffffu, at, 31) + x - nk;
            if (at + nk <= CAP) {
                Key* d = S.keys + at;
                Roll<W> roll;
                roll.start(rec, k);
                for (uint32_t t = 0; t < nk; ++t) {
                    *d++ = roll.key(k);
                    roll.step(k);
                }
                if (w > 1)
                    for (uint32_t t = 0; t < nk; ++t) S.cnt[at + t] = w - 1;
            }
            __syncwarp();
        };
        if (W == 1 && dedup) {
#pragma unroll
            for (uint32_t j = 0; j < DM; ++j)
                if (j * COUNT_THREADS + (tid & ~31u) < nrec) unpack(mine[j], weight[j] ? mine[j].n() : 0, weight[j]);
        } else {
            for (uint32_t i = tid; (i & ~31u) < nrec; i += COUNT_THREADS) {
                const Rec<W> rec = ahead;
                if ((i & ~31u) + COUNT_THREADS < nrec) ahead = load_at(g, i + COUNT_THREADS);
                unpack(rec, rec.n(), 1);
            }
        }
        __syncthreads();
        const uint32_t n = min(S.staged, CAP);
        ahead = load_at(S.grp[q == 2 ? 0 : q + 1], tid);
        uint32_t newm = 0, pend = 0;
        // A CAS per key at its home slot, and one at the next slot of its probe if the
        // home slot holds another key; the few keys (1.5 % in a table a quarter full)
        // that both find taken stay pending (bit u of pend).
#pragma unroll 1
        for (uint32_t u0 = 0; u0 * COUNT_THREADS < n; u0 += U) {
            Key K[U];
            uint32_t en[U], h[U], e[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const uint32_t i = (u0 + u) * COUNT_THREADS + tid;
                K[u] = S.keys[i];
                place_of<W>(slot_hash(K[u]), i, h[u], en[u]);
                e[u] = IDX_MASK;  // no key: nothing below happens
                if (i < n) e[u] = atomicCAS(&S.table[h[u]], NO_ENTRY, en[u]);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const uint32_t bit = 1u << (u0 + u);
                uint32_t f = e[u];
                if (f == NO_ENTRY) newm |= bit;
                if (f < NO_ENTRY && f != IDX_MASK) {
                    if (((f ^ en[u]) >> IDX_BITS) != 0 || !O::eq(S.keys[f & IDX_MASK], K[u])) {
                        f = atomicCAS(&S.table[next_slot<W>(h[u], en[u])], NO_ENTRY, en[u]);
                        if (f == NO_ENTRY) newm |= bit;
                        else if (((f ^ en[u]) >> IDX_BITS) != 0 || !O::eq(S.keys[f & IDX_MASK], K[u])) { pend |= bit; f = NO_ENTRY; }
                    }
                    if (f != NO_ENTRY) {  // known: its weight to the place that came first
                        const uint32_t i = (u0 + u) * COUNT_THREADS + tid, w = S.cnt[i];
                        atomicAdd(&S.cnt[f & IDX_MASK], w + 1);
                        if (w) S.cnt[i] = 0;
                    }
                }
            }
        }
        while (pend) {
            const uint32_t bit = pend & (0u - pend), i = (31 - __clz(bit)) * COUNT_THREADS + tid;
            pend ^= bit;
            const Key key = S.keys[i];
            uint32_t h, en;
            place_of<W>(slot_hash(key), i, h, en);
            h = next_slot<W>(h, en);
            for (uint32_t p = 0; p < SLOTS; ++p) {
                h = next_slot<W>(h, en);
                const uint32_t e = atomicCAS(&S.table[h], NO_ENTRY, en);
                if (e == NO_ENTRY) { newm |= bit; break; }
                if (((e ^ en) >> IDX_BITS) == 0 && O::eq(S.keys[e & IDX_MASK], key)) {
                    const uint32_t w = S.cnt[i];
                    atomicAdd(&S.cnt[e & IDX_MASK], w + 1);
                    if (w) S.cnt[i] = 0;
                    break;
                }
            }
        }
        __syncwarp();
        write_out<W>(P, S, n, newm, sample, distinct, [&] {
            if (tid == 0) {  // group g + 3's entry into slot q, the index after it claimed
                S.staged = 0;
                if (!dedup && S.dedup) --S.dedup;
                copy_group(&S.grp[q], P, S.pending, g_end);
                S.pending = P.g_begin + atomicAdd(P.work, 1ull);
            }
        });
        if (tid == 0) asm volatile("cp.async.wait_all;" ::: "memory");  // group g + 3's entry has landed
        __syncthreads();  // the store may be filled again
    }
    if (lane == 0 && distinct) atomicAdd(&P.ctr[P2C_DISTINCT], (unsigned long long)distinct);
}

// ---------------------------------------------------------------- larger groups
// Inserts the staged keys of places [n, m); those that another came before are holes.
template <int W>
__device__ __forceinline__ void insert_staged(CountSmem<W>& S, uint32_t n, uint32_t m, uint32_t& newm) {
    using O = KeyOps<W>;
    using Key = typename O::Key;
    constexpr uint32_t SLOTS = CountSmem<W>::SLOTS;
    const uint32_t tid = threadIdx.x;
    for (uint32_t u = n / COUNT_THREADS; u * COUNT_THREADS < m; ++u) {
        const uint32_t i = u * COUNT_THREADS + tid;
        if (i < n || i >= m) continue;
        const Key key = S.keys[i];
        uint32_t h, en;
        place_of<W>(slot_hash(key), i, h, en);
        for (uint32_t p = 0; p < SLOTS; ++p) {
            const uint32_t e = atomicCAS(&S.table[h], NO_ENTRY, en);
            if (e == NO_ENTRY) { newm |= 1u << u; break; }
            if (((e ^ en) >> IDX_BITS) == 0 && O::eq(S.keys[e & IDX_MASK], key)) {
                // only this thread reads or clears the count of a place that is in no entry
                atomicAdd(&S.cnt[e & IDX_MASK], S.cnt[i] + 1);
                S.cnt[i] = 0;
                break;
            }
            h = next_slot<W>(h, en);
        }
    }
}

// True, and the key's count up by weight, if the store holds the key.
template <int W>
__device__ __forceinline__ bool count_known(CountSmem<W>& S, const typename KeyOps<W>::Key& key, uint32_t weight) {
    uint32_t h, en;
    place_of<W>(slot_hash(key), 0, h, en);
    for (uint32_t p = 0; p < CountSmem<W>::SLOTS; ++p) {
        const uint32_t e = *(const volatile uint32_t*)&S.table[h];
        if (e == NO_ENTRY) return false;
        if (((e ^ en) >> IDX_BITS) == 0 && KeyOps<W>::eq(S.keys[e & IDX_MASK], key)) {
            atomicAdd(&S.cnt[e & IDX_MASK], weight);
            return true;
        }
        h = next_slot<W>(h, en);
    }
    return false;
}

// Every lane of the warp calls it: lanes with a get consecutive places from *at on.
__device__ __forceinline__ uint32_t warp_place(uint32_t* at, bool a, unsigned peers) {
    uint32_t base = 0;
    const uint32_t lane = threadIdx.x & 31;
    const int lead = __ffs(peers) - 1;
    if (a && (int)lane == lead) base = atomicAdd(at, (uint32_t)__popc(peers));
    base = __shfl_sync(0xffffffffu, base, lead < 0 ? 0 : lead);
    return base + __popc(peers & ((1u << lane) - 1));
}

// The next records of a range in rounds. A round looks its keys up first: the
// ones that the store holds are counted (equal records of a warp, a repeat's, as
// one of their number), only the others are staged behind the store's keys and
// inserted; those that another of the round came before stay as holes. The first
// round is short, since all of its keys are staged. Takes records [r, nrec) until
// they are all counted or the store is 7/8 full and returns how far it came; n:
// places in use, newm: bit u set if this thread's place u * COUNT_THREADS + threadIdx.x
// holds a new key. Every thread of the CTA calls it; ends with a barrier.
template <int W>
__device__ __forceinline__ unsigned long long count_rounds(const CountParams& P, CountSmem<W>& S,
                                                           unsigned long long lo, unsigned long long r,
                                                           unsigned long long nrec, uint32_t parts, uint32_t part,
                                                           uint32_t& n, uint32_t& newm) {
    using Key = typename KeyOps<W>::Key;
    constexpr uint32_t CAP = CountShape<W>::CAP;
    const uint32_t tid = threadIdx.x, lane = tid & 31;
    const int k = P.k;
    while (r < nrec && CAP - n >= CAP / 8) {
        // as many records as fit if all of their keys are new; the warps share them evenly
        const uint32_t take = (uint32_t)min((unsigned long long)((n ? CAP - n : 512u) / REC_MAX), nrec - r);
        const uint32_t per = (take + COUNT_THREADS / 32 - 1) / (COUNT_THREADS / 32), w0 = (tid >> 5) * per;
        const uint32_t w1 = min(w0 + per, take);
        for (uint32_t i0 = w0; i0 < w1; i0 += 32) {
            Rec<W> c;
            uint32_t nk = 0;
            if (i0 + lane < w1) {
                c = load_rec<W>(P.recs, lo + r + i0 + lane);
                nk = c.n();
            }
            unsigned same = __match_any_sync(0xffffffffu, nk ? c.w[0] : (unsigned long long)lane);
            same &= __match_any_sync(0xffffffffu, nk ? c.w[1] : ~(unsigned long long)lane);
            if constexpr (W == 2) {
                same &= __match_any_sync(0xffffffffu, nk ? c.w[2] : (unsigned long long)lane);
                same &= __match_any_sync(0xffffffffu, nk ? c.w[3] : ~(unsigned long long)lane);
            }
            const uint32_t weight = __popc(same);
            if (lane != (uint32_t)__ffs(same) - 1) nk = 0;
            const uint32_t steps = __reduce_max_sync(0xffffffffu, nk);
            Roll<W> roll;
            if (nk) roll.start(c, k);
            for (uint32_t t = 0; t < steps; ++t) {
                bool a = t < nk;
                Key key;
                if (a) {
                    key = roll.key(k);
                    roll.step(k);
                    a = parts == 1 || key_part<W>(key, parts) == part;
                }
                if (a && count_known<W>(S, key, weight)) a = false;
                const unsigned bal = __ballot_sync(0xffffffffu, a);
                uint32_t base = 0;
                if (lane == 0 && bal) base = atomicAdd(&S.staged, (uint32_t)__popc(bal));
                base = n + __shfl_sync(0xffffffffu, base, 0) + __popc(bal & ((1u << lane) - 1));
                if (a && base < CAP) {
                    S.keys[base] = key;
                    S.cnt[base] = weight - 1;
                }
            }
        }
        __syncthreads();
        const uint32_t m = min(n + S.staged, CAP);
        insert_staged<W>(S, n, m, newm);
        __syncthreads();  // the round is in the table; every thread has its size
        if (tid == 0) S.staged = 0;
        n = m;
        r += take;
        __syncthreads();
    }
    return r;
}

// A group of more distinct k-mers than a store holds, counted as F key-hash parts: its
// k-mers are unpacked twice, to count each part's and to write them, part by part, to
// this CTA's room in global memory (which stays in L2); then each part goes through the
// store. A part that does not fit after all comes back through the retry list. (As F
// passes over the records instead, each unpacking all and keeping its own part's:
// 1.5 Gbp with k=27 m=15, whose hash has few values, took 264 ms to count against 40.)
template <int W>
__device__ __forceinline__ void split_group(const CountParams& P, CountSmem<W>& S, const Group& g, uint32_t F,
                                            uint32_t& distinct) {
    using Key = typename KeyOps<W>::Key;
    constexpr uint32_t CAP = CountShape<W>::CAP;
    const uint32_t tid = threadIdx.x, lane = tid & 31;
    const int k = P.k;
    Key* buf = static_cast<Key*>(P.split) + (size_t)blockIdx.x * BIG_KEYS;
    const uint32_t nrec = (uint32_t)(g.hi - g.lo);
    if (tid < MAX_SPLIT) S.part_end[tid] = 0;
    __syncthreads();
    for (int pass = 0; pass < 2; ++pass) {
        for (uint32_t i0 = tid - lane; i0 < nrec; i0 += COUNT_THREADS) {
            Rec<W> c;
            uint32_t nk = 0;
            if (i0 + lane < nrec) {
                c = load_rec<W>(P.recs, g.lo + i0 + lane);
                nk = c.n();
            }
            const uint32_t steps = __reduce_max_sync(0xffffffffu, nk);
            Roll<W> roll;
            if (nk) roll.start(c, k);
            for (uint32_t t = 0; t < steps; ++t) {
                const bool a = t < nk;
                Key key;
                uint32_t p = 0;
                if (a) {
                    key = roll.key(k);
                    roll.step(k);
                    p = key_part<W>(key, F);
                }
                // the warp's lanes of the same part
                unsigned peers = __ballot_sync(0xffffffffu, a);
                for (uint32_t b = 1; b < F; b <<= 1) {
                    const unsigned s = __ballot_sync(0xffffffffu, p & b);
                    peers &= p & b ? s : ~s;
                }
                if (pass == 0) {
                    if (a && (int)lane == __ffs(peers) - 1) atomicAdd(&S.part_end[p], (uint32_t)__popc(peers));
                } else {
                    const uint32_t at = warp_place(&S.part_end[p], a, a ? peers : 0u);
                    if (a && at < BIG_KEYS) buf[at] = key;
                }
            }
        }
        __syncthreads();
        if (pass == 0 && tid < MAX_SPLIT) {  // the parts' first places, by a scan of one warp
            const uint32_t v = S.part_end[tid];
            uint32_t x = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
                if ((int)tid >= o) x += y;
            }
            S.part_end[tid] = x - v;
        }
        __syncthreads();
    }
    for (uint32_t p = 0; p < F; ++p) {
        const uint32_t end = min(S.part_end[p], BIG_KEYS);
        uint32_t r = p ? S.part_end[p - 1] : 0, n = 0, newm = 0;
        while (r < end && CAP - n >= CAP / 8) {
            // all of the part if its k-mers fit; else few at first, since all of those take places
            const uint32_t take = min(n ? CAP - n : (end - r <= CAP ? CAP : 512u), end - r);
            uint32_t m = take;
            if (n == 0) {  // the store is empty
                for (uint32_t i = tid; i < take; i += COUNT_THREADS) S.keys[i] = buf[r + i];
                __syncthreads();
            } else {
                for (uint32_t i0 = tid - lane; i0 < take; i0 += COUNT_THREADS) {
                    bool a = i0 + lane < take;
                    Key key;
                    if (a) {
                        key = buf[r + i0 + lane];
                        a = !count_known<W>(S, key, 1);
                    }
                    const unsigned bal = __ballot_sync(0xffffffffu, a);
                    const uint32_t at = n + warp_place(&S.staged, a, bal);
                    if (a && at < CAP) S.keys[at] = key;
                }
                __syncthreads();
                m = min(n + S.staged, CAP);
            }
            insert_staged<W>(S, n, m, newm);
            __syncthreads();
            if (tid == 0) S.staged = 0;
            n = m;
            r += take;
            __syncthreads();
        }
        if (r < end) {
            if (tid == 0) {
                Group f = g;
                f.parts = 2 * F;
                const unsigned long long i = atomicAdd(P.n_retry, 2ull);
                if (i + 1 < P.retry_cap)
                    for (uint32_t q = 0; q < 2; ++q) {
                        f.part = p + q * F;
                        P.retry[i + q] = f;
                    }
            }
            for (uint32_t i = tid; i < n; i += COUNT_THREADS) S.cnt[i] = 0;
            clear_table<W>(S);
        } else if (n) {
            write_out<W>(P, S, n, newm, g.sample, distinct, [] {});
        }
        __syncthreads();
    }
}

// Groups of more than CAP and at most BIG_KEYS k-mers (one bin each), and key-hash parts
// of such groups, one CTA each. A group whose distinct keys do not fit is split
// (split_group) or, without room for that (a job below SPLIT_MIN, one with a memory
// budget), comes back as F key-hash parts, F the power of two that gives half-full
// stores for the places estimated from the share of the group seen; past MAX_PARTS
// parts it goes to the global-memory table.
template <int W>
__global__ void __launch_bounds__(COUNT_THREADS, COUNT_PER_SM) k_rounds(const __grid_constant__ CountParams P) {
    constexpr uint32_t CAP = CountShape<W>::CAP;
    extern __shared__ __align__(128) uint8_t smem[];
    CountSmem<W>& S = *reinterpret_cast<CountSmem<W>*>(smem);
    const uint32_t tid = threadIdx.x;
    uint32_t distinct = 0;
    const unsigned long long g_end = list_end(P);
    if (P.g_begin + blockIdx.x >= g_end) return;
    start_store<W>(S);
    // groups differ in size by more than ten: taken from a counter, the first of each CTA aside
    for (unsigned long long gi = P.g_begin + blockIdx.x; gi < g_end; gi = S.pending) {
        __syncthreads();
        if (tid == 0) S.pending = P.g_begin + gridDim.x + atomicAdd(P.work, 1ull);
        const Group g = P.list[gi];
        const unsigned long long nrec = g.hi - g.lo;
        uint32_t n = 0, newm = 0;
        // a group that may be split: its first eighth tells whether that is needed
        const bool may = P.split && g.parts == 1 && g.keys > CAP && g.keys <= BIG_KEYS;
        const unsigned long long probe = may ? nrec / 8 + 1 : nrec;
        unsigned long long r = 0, to = probe;
        uint64_t est = 0;
        for (;;) {
            r = count_rounds<W>(P, S, g.lo, r, to, g.parts, g.part, n, newm);
            est = (uint64_t)n * nrec / r;
            if (r < to || to == nrec || est > CAP) break;
            to = nrec;
        }
        if (r < nrec && may) {  // too many distinct keys
            for (uint32_t i = tid; i < n; i += COUNT_THREADS) S.cnt[i] = 0;
            clear_table<W>(S);
            uint32_t F = 2;
            while (F < MAX_SPLIT && (uint64_t)F * (CAP / 4 * 3) < est) F <<= 1;
            split_group<W>(P, S, g, F, distinct);  // ends with a barrier
            continue;
        }
        if (r < nrec) {
            if (tid == 0) {
                Group f = g;
                if (g.parts < MAX_PARTS) {
                    const uint64_t need = ((uint64_t)n * nrec / r + CAP / 2 - 1) / (CAP / 2);
                    uint32_t F = 2;
                    while (F < need) F <<= 1;
                    while (g.parts * F > MAX_PARTS) F >>= 1;
                    const unsigned long long i = atomicAdd(P.n_retry, (unsigned long long)F);
                    f.parts = F * g.parts;
                    if (i + F - 1 < P.retry_cap)
                        for (uint32_t j = 0; j < F; ++j) {
                            f.part = g.part + j * g.parts;
                            P.retry[i + j] = f;
                        }
                } else {
                    const unsigned long long i = atomicAdd(&P.ctr[P2C_FALLBACK], 1ull);
                    if (i < P.fallback_cap) P.fallback[i] = f;
                }
            }
            for (uint32_t i = tid; i < n; i += COUNT_THREADS) S.cnt[i] = 0;
            clear_table<W>(S);
        } else {
            write_out<W>(P, S, n, newm, g.sample, distinct, [] {});
        }
        __syncthreads();
    }
    if ((tid & 31) == 0 && distinct) atomicAdd(&P.ctr[P2C_DISTINCT], (unsigned long long)distinct);
}

// Groups of more than BIG_KEYS k-mers (one bin: a repeat's, or one conserved
// minimizer's), each shared by many CTAs: blockIdx.y picks the group, the CTAs of a row
// its chunks of BIG_CHUNK records. A chunk's keys are counted in the CTA's own store as
// above, and the store's (key, count) pairs added to a table in global memory whenever it
// fills up and at the end, so a k-mer that the group repeats costs a global atomic per
// store, not per instance.
template <int W>
__global__ void __launch_bounds__(COUNT_THREADS, COUNT_PER_SM)
    k_big(const __grid_constant__ CountParams P, const __grid_constant__ FallbackParams F) {
    using Key = typename KeyOps<W>::Key;
    extern __shared__ __align__(128) uint8_t smem[];
    CountSmem<W>& S = *reinterpret_cast<CountSmem<W>*>(smem);
    const uint32_t tid = threadIdx.x;
    start_store<W>(S);
    __syncthreads();
    const Group g = P.list[P.g_begin + blockIdx.y];
    const unsigned long long nrec = g.hi - g.lo;
    for (unsigned long long c = (unsigned long long)blockIdx.x * BIG_CHUNK; c < nrec; c += (unsigned long long)gridDim.x * BIG_CHUNK) {
        const unsigned long long end = min(nrec, c + BIG_CHUNK);
        for (unsigned long long r = c; r < end;) {
            uint32_t n = 0, newm = 0;
            r = count_rounds<W>(P, S, g.lo, r, end, 1, 0, n, newm);
            for (uint32_t u = 0; u * COUNT_THREADS < n; ++u) {
                const uint32_t i = u * COUNT_THREADS + tid;
                if ((newm >> u) & 1u)
                    if (!tbl_add<W>(static_cast<Key*>(F.tkeys), F.tcnt, F.mask, S.keys[i], S.cnt[i] + 1, F.mask))
                        atomicExch(F.fail, 1u);
                if (i < n) S.cnt[i] = 0;
            }
            clear_table<W>(S);
            __syncthreads();
        }
    }
}

// ---------------------------------------------------------------- fallback
// A key range (one key-hash part of it) that did not fit in shared memory,
// counted in a global table of S slots (power of two >= 2 x the range).
template <int W>
__global__ void k_fb_insert(FallbackParams F) {
    using O = KeyOps<W>;
    auto* tk = reinterpret_cast<typename O::Key*>(F.tkeys);
    for (unsigned long long i = F.lo + (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < F.hi;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const Rec<W> c = load_rec<W>(F.recs, i);
        const uint32_t n = c.n();
        Roll<W> roll;
        roll.start(c, F.k);
        for (uint32_t t = 0; t < n; ++t, roll.step(F.k)) {
            const typename O::Key key = roll.key(F.k);
            if (key_part<W>(key, F.parts) != F.part) continue;
            if (!tbl_add<W>(tk, F.tcnt, F.mask, key, 1, F.mask)) atomicExch(F.fail, 1u);
        }
    }
}

template <int W>
__global__ void k_fb_init(void* keys, uint32_t* cnt, uint64_t S) {
    using O = KeyOps<W>;
    auto* kk = reinterpret_cast<typename O::Key*>(keys);
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < S; i += (uint64_t)gridDim.x * blockDim.x) {
        kk[i] = O::empty();
        cnt[i] = 0;
    }
}

// Write the occupied slots that pass ci/cx. A warp takes EXTRACT slots of each lane at a
// time, with one output atomic for them: with one per 32 slots the counter was what
// bound it (2^28 slots: 6.4 ms, 2.2 now).
constexpr int EXTRACT = 8;
template <int W>
__global__ void __launch_bounds__(256) k_fb_extract(const void* keys, const uint32_t* cnt, uint64_t S,
                                                    CountParams P, uint32_t sample) {
    using Key = typename KeyOps<W>::Key;
    const Key* kk = static_cast<const Key*>(keys);
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t warps = (uint64_t)gridDim.x * (blockDim.x / 32);
    const uint64_t warp = (uint64_t)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
    unsigned long long distinct = 0;
    for (uint64_t s0 = warp * (32 * EXTRACT); s0 < S; s0 += warps * (32 * EXTRACT)) {  // S: a multiple of 256
        Key key[EXTRACT];
        uint32_t c[EXTRACT], kept = 0, mine = 0;
#pragma unroll
        for (int u = 0; u < EXTRACT; ++u) {
            key[u] = kk[s0 + u * 32 + lane];
            c[u] = cnt[s0 + u * 32 + lane];
        }
#pragma unroll
        for (int u = 0; u < EXTRACT; ++u) {
            const bool has = !KeyOps<W>::is_empty(key[u]);
            distinct += has;
            if (has && c[u] >= P.ci && c[u] <= P.cx) {
                kept |= 1u << u;
                ++mine;
            }
        }
        uint32_t at = mine;  // exclusive scan over the lanes
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, at, o);
            if ((int)lane >= o) at += y;
        }
        const uint32_t all = __shfl_sync(0xffffffffu, at, 31);
        if (!all) continue;
        at -= mine;
        unsigned long long base = 0;
        if (lane == 0) {
            base = atomicAdd(&P.ctr[P2C_OUT], (unsigned long long)all);
            if (P.sample_tot) atomicAdd(&P.sample_tot[sample], all);
        }
        base = __shfl_sync(0xffffffffu, base, 0) + at;
#pragma unroll
        for (int u = 0; u < EXTRACT; ++u)
            if ((kept >> u) & 1u) {
                if (base < P.out_cap) {
                    KeyOps<W>::store(P.out_keys, base, key[u]);
                    P.out_counts[base] = c[u];
                    if (P.out_sample) P.out_sample[base] = sample;
                }
                ++base;
            }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) distinct += __shfl_down_sync(0xffffffffu, distinct, o);
    if (lane == 0 && distinct) atomicAdd(&P.ctr[P2C_DISTINCT], distinct);
}

// ---------------------------------------------------------------- sample-major output
// Jobs of several samples: the pairs, in group order, go sample-major so that
// each sample's pairs are one range (the counting kernels add up the samples'
// totals). The pairs that a counting warp wrote are contiguous and of one sample,
// so the 128 pairs that a warp takes here at a time nearly always share it: one
// atomic for them, else one per sample in each 32 (match_any).
constexpr int SAMP_UNROLL = 4;
template <int W>
__global__ void __launch_bounds__(256) k_samp_scatter(const void* __restrict__ keys, const uint32_t* __restrict__ cnt,
                                                      const uint32_t* __restrict__ samp, uint64_t n,
                                                      unsigned long long* __restrict__ cur, void* __restrict__ keys2,
                                                      uint32_t* __restrict__ cnt2) {
    using O = KeyOps<W>;
    const uint32_t lane = threadIdx.x & 31;
    const auto* kk = static_cast<const typename O::Key*>(keys);
    const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5, warps = (uint64_t)gridDim.x * blockDim.x >> 5;
    for (uint64_t i0 = warp * 32 * SAMP_UNROLL; i0 < n; i0 += warps * 32 * SAMP_UNROLL) {
        uint32_t s[SAMP_UNROLL], c[SAMP_UNROLL];
        typename O::Key k[SAMP_UNROLL];
        const uint32_t m = (uint32_t)min((uint64_t)(32 * SAMP_UNROLL), n - i0);
        bool one = true;
#pragma unroll
        for (int u = 0; u < SAMP_UNROLL; ++u) {
            const uint32_t j = 32 * u + lane;
            s[u] = 0xFFFFFFFFu;
            if (j < m) {
                s[u] = samp[i0 + j];
                k[u] = kk[i0 + j];
                c[u] = cnt[i0 + j];
            }
        }
        const uint32_t first = __shfl_sync(0xffffffffu, s[0], 0);
#pragma unroll
        for (int u = 0; u < SAMP_UNROLL; ++u) one = one && (s[u] == first || 32 * u + lane >= m);
        one = __all_sync(0xffffffffu, one);
        unsigned long long base = 0;
        if (one && lane == 0) base = atomicAdd(&cur[first], (unsigned long long)m);
        base = __shfl_sync(0xffffffffu, base, 0);
#pragma unroll
        for (int u = 0; u < SAMP_UNROLL; ++u) {
            uint64_t o = base + 32 * u + lane;
            if (!one) {
                const unsigned peers = __match_any_sync(0xffffffffu, s[u]);
                const uint32_t leader = __ffs(peers) - 1;
                unsigned long long b = 0;
                if (s[u] != 0xFFFFFFFFu && lane == leader) b = atomicAdd(&cur[s[u]], (unsigned long long)__popc(peers));
                o = __shfl_sync(0xffffffffu, b, leader) + __popc(peers & ((1u << lane) - 1));
            }
            if (32 * u + lane < m) {
                O::store(keys2, o, k[u]);
                cnt2[o] = c[u];
            }
        }
    }
}

// ---------------------------------------------------------------- host side
size_t key_bytes(int W) { return W == 1 ? 8 : 16; }

uint64_t table_slots(uint64_t n, int k) {
    if (k < 32) n = std::min<uint64_t>(n, 1ull << (2 * k));
    if (n >= 1ull << 31) return 0;
    uint64_t S = 1024;
    while (S < 2 * n + 2) S <<= 1;
    return S;
}

uint32_t count_slots(int) { return 8192; }

uint32_t group_keys(int W, uint32_t pct) {
    const uint32_t cap = W == 1 ? CountShape<1>::CAP : CountShape<2>::CAP;
    return std::max<uint32_t>(1, std::min(count_slots(W) * pct / 100, cap));
}

// Keys that k_plan puts in a group.
static uint32_t group_target(const P2Input& in) {
    const uint32_t t = group_keys(in.W, in.group_pct);
    // jobs too small for a full group per CTA: smaller groups, so that more SMs count
    const uint64_t share = in.n_kmers / (COUNT_PER_SM * (uint64_t)std::max<uint32_t>(1, in.n_sm));
    return (uint32_t)std::min<uint64_t>(t, std::max<uint64_t>(COUNT_THREADS, share));
}

namespace {
struct Carve {
    uint8_t* base;
    size_t off, cap;
    bool ok;
    template <class T>
    T* take(size_t n) {
        off = (off + 255) & ~size_t(255);
        if (off + n * sizeof(T) > cap) { ok = false; return nullptr; }
        T* p = reinterpret_cast<T*>(base + off);
        off += n * sizeof(T);
        return p;
    }
};

struct P2Plan {
    uint64_t groups_cap = 0, retry_cap = 0, nsum = 0;
};

// Warps of k_plan per segment. Its steps are serial within a warp (one group
// each, about a microsecond of dependent reads), so long segments are shared out
// until a share has about 32 groups (8 in a small job, where the steps count most);
// fewer would leave more of the last groups of the shares half filled.
uint32_t plan_split(const P2Input& in) {
    uint32_t s = 1;
    const uint64_t groups = in.deferred ? 8 : 32;
    while (s < 64 && in.n_kmers / ((uint64_t)in.n_segs * 2 * s + 1) > groups * group_target(in)) s *= 2;
    return s;
}

P2Plan make_plan(const P2Input& in) {
    P2Plan L;
    // a segment of K keys has fewer than 2 K / target + 1 groups (two neighbouring
    // groups of k_plan hold more than `target` keys together)
    const uint64_t target = group_target(in);
    L.groups_cap = 2 * in.n_kmers / target + (uint64_t)in.n_segs * plan_split(in) + 1;
    L.retry_cap = std::max<uint64_t>(4096, 2 * L.groups_cap);
    L.nsum = scan_scratch(std::max<uint64_t>(in.all_bins, in.n_samples));
    return L;
}

// The scratch regions of one run, in order (the same walk sizes and places them).
struct P2Regions {
    unsigned long long* ctr;
    unsigned long long* aux;  // [0..1] retry counters
    unsigned long long* work; // [0..15] group counters of k_count's launches, [16] k_rounds'
    unsigned long long* kofs;
    unsigned long long* rofs;
    uint32_t* gfirst;
    unsigned long long* sums;
    Segment* segs;
    Group* normal;
    Group* heavy;
    Group* big;
    Group* retry[2];
    Group* fb;
    unsigned long long* scur;  // [n_samples] cursors of the sample-major copy
    uint32_t* stot;            // [n_samples] pairs of each sample
    uint8_t* recs;
    uint8_t* split;            // [k_rounds' CTAs][BIG_KEYS] keys, or null
};

// CTAs of k_rounds with room for splitting: as many as there can be groups for.
uint64_t split_ctas(const P2Input& in) {
    if (!in.roomy || in.n_kmers < SPLIT_MIN) return 0;
    return std::min<uint64_t>((uint64_t)in.n_sm * COUNT_PER_SM, in.n_kmers / CountShape<2>::CAP + 1);
}

P2Regions carve(Carve& c, const P2Input& in, const P2Plan& L) {
    P2Regions R;
    R.ctr = c.take<unsigned long long>(P2C_COUNT);
    R.aux = c.take<unsigned long long>(2);
    R.work = c.take<unsigned long long>(17);
    R.kofs = c.take<unsigned long long>((size_t)in.all_bins + 1);
    R.rofs = c.take<unsigned long long>((size_t)in.all_bins + 1);
    R.gfirst = c.take<uint32_t>(in.all_bins);
    R.sums = c.take<unsigned long long>(L.nsum);
    R.segs = c.take<Segment>(in.n_segs + 1);
    R.normal = c.take<Group>(L.groups_cap);
    R.heavy = c.take<Group>(L.groups_cap);
    R.big = c.take<Group>(in.n_kmers / BIG_KEYS + 1);
    R.retry[0] = c.take<Group>(L.retry_cap);
    R.retry[1] = c.take<Group>(L.retry_cap);
    R.fb = c.take<Group>(FALLBACK_CAP);
    R.scur = c.take<unsigned long long>(in.n_samples + 1);
    R.stot = c.take<uint32_t>(in.n_samples + 1);
    R.recs = c.take<uint8_t>((in.n_recs + 1) * 16 * (size_t)in.W);
    const uint64_t sc = split_ctas(in);
    R.split = sc ? c.take<uint8_t>(sc * BIG_KEYS * key_bytes(in.W)) : nullptr;
    return R;
}
}  // namespace

// The work that goes with every bin (histogram, scan, plan) is small next to the
// keys', and bins of a few hundred keys pack into groups with little left over:
// about 512 stream bytes per bin, up to 2^22 bins. (3.1 Gbp in 2^20 bins of 2,950
// k-mers filled groups of 4,096 to 72 %; small calls spent most of their time on
// 2^20 empty bins.)
int job_bin_bits(uint64_t n, uint32_t n_samples, uint32_t seg_bits) {
    const int most = n < (1ull << 34) ? MAX_BIN_BITS : BIN_BITS;
    int b = std::max<int>(8, (int)seg_bits);
    while ((2ull << b) <= n / 256 && b < most) ++b;
    while (b < BIN_BITS && (1ull << b) < 4ull * n_samples) ++b;
    return b;
}

SampleBins layout_bins(const std::vector<unsigned long long>& sample_start, uint32_t seg_bins, int bin_bits) {
    const uint32_t all = 1u << bin_bits;
    SampleBins B;
    B.start = sample_start;
    const size_t n = sample_start.size() - 1;
    const double total = (double)std::max<unsigned long long>(1, sample_start[n] - sample_start[0]);
    B.base.resize(n);
    B.bits.resize(n);
    // 2^bits <= the sample's share of `budget` bins (at least one bin)
    auto assign = [&](double budget) {
        uint64_t used = 0;
        for (size_t i = 0; i < n; ++i) {
            const double share = budget * (double)(sample_start[i + 1] - sample_start[i]) / total;
            uint32_t b = 0;
            while (b < (uint32_t)bin_bits && (double)(2ull << b) <= share) ++b;
            B.bits[i] = (uint8_t)b;
            B.base[i] = (uint32_t)used;
            used += 1ull << b;
        }
        return used;
    };
    if (assign((double)all) > all) assign((double)(all - n));  // one bin set aside per sample
    seg_bins = std::max<uint32_t>(1, seg_bins);
    for (size_t i = 0; i < n; ++i) {
        const uint32_t hi = B.base[i] + (1u << B.bits[i]);
        for (uint32_t lo = B.base[i]; lo < hi; lo += seg_bins) {
            Segment sg;
            sg.bin_lo = lo;
            sg.bin_hi = std::min(hi, lo + seg_bins);
            sg.sample = (uint32_t)i;
            sg.pad = 0;
            B.segs.push_back(sg);
        }
    }
    return B;
}

size_t phase2_scratch_bytes(const P2Input& in) {
    const P2Plan L = make_plan(in);
    Carve c{nullptr, 0, ~size_t(0), true};
    carve(c, in, L);
    return c.off + 256;
}

#define P2_CK(call, what)                                            \
    do {                                                             \
        cudaError_t e_ = (call);                                     \
        if (e_ != cudaSuccess) {                                     \
            err = std::string(what) + ": " + cudaGetErrorString(e_); \
            return TG_ERR_CUDA;                                      \
        }                                                            \
    } while (0)

// Small counter reads (see OVERLAP_WORDS): up to three ranges to the mapped host
// words dst (device address), fenced for the host.
struct PeekRange {
    const unsigned long long* p;
    uint32_t n;
};
__global__ void k_peek(PeekRange a, PeekRange b, PeekRange c, unsigned long long* dst) {
    const uint32_t i = threadIdx.x;
    if (i < a.n) dst[i] = a.p[i];
    else if (i < a.n + b.n) dst[i] = b.p[i - a.n];
    else if (i < a.n + b.n + c.n) dst[i] = c.p[i - a.n - b.n];
    __threadfence_system();
}

cudaError_t launch_peek(const unsigned long long* src, uint32_t n, unsigned long long* dst, cudaStream_t st) {
    k_peek<<<1, 32, 0, st>>>({src, n}, {}, {}, dst);
    return cudaGetLastError();
}

// Reads the ranges into out (host), one after the other, then waits for the
// stream. With mapped words (ov.wave_out_dev) a kernel stores them there;
// otherwise cudaMemcpyAsync.
static cudaError_t read_counters(const P2Overlap& ov, PeekRange a, PeekRange b, PeekRange c, unsigned long long* out,
                                 cudaStream_t st) {
    const uint32_t n = a.n + b.n + c.n;
    if (ov.wave_out && ov.wave_out_dev && n <= 32) {
        k_peek<<<1, 32, 0, st>>>(a, b, c, ov.wave_out_dev + 16);
        cudaError_t e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) return e;
        const volatile unsigned long long* w = ov.wave_out + 16;
        for (uint32_t i = 0; i < n; ++i) out[i] = w[i];
        return cudaSuccess;
    }
    cudaError_t e = cudaSuccess;
    for (const PeekRange& r : {a, b, c}) {
        if (e == cudaSuccess && r.n) e = cudaMemcpyAsync(out, r.p, 8 * (size_t)r.n, cudaMemcpyDeviceToHost, st);
        out += r.n;
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    return e;
}

// Before phase 2, in one launch: its counters at zero and, for a job of one sample,
// whose segments are equal runs of its bins, the segments (no copy from pageable
// memory, which the host waits for).
__global__ void __launch_bounds__(256) k_setup(unsigned long long* ctr, uint32_t n_ctr, Segment* segs, uint32_t n,
                                               uint32_t lo, uint32_t per, uint32_t sample) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
    for (uint32_t i = t; i < n_ctr; i += stride) ctr[i] = 0;
    for (uint32_t i = t; i < n; i += stride) {
        Segment s;
        s.bin_lo = lo + i * per;
        s.bin_hi = s.bin_lo + per;
        s.sample = sample;
        s.pad = 0;
        segs[i] = s;
    }
}

static cudaError_t setup(const P2Input& in, const P2Regions& R, cudaStream_t st) {
    const Segment f = in.n_segs ? in.segs[0] : Segment{};
    const uint32_t per = f.bin_hi - f.bin_lo;
    bool equal = true;
    for (uint32_t i = 0; i < in.n_segs && equal; ++i)
        equal = in.segs[i].sample == f.sample && in.segs[i].bin_lo == f.bin_lo + i * per &&
                in.segs[i].bin_hi == f.bin_lo + (i + 1) * per;
    // ctr, aux and work lie one after the other
    k_setup<<<2, 256, 0, st>>>(R.ctr, (uint32_t)(R.work + 16 - R.ctr), R.segs, equal ? in.n_segs : 0, f.bin_lo, per, f.sample);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess && !equal)
        e = cudaMemcpyAsync(R.segs, in.segs, (size_t)in.n_segs * sizeof(Segment), cudaMemcpyHostToDevice, st);
    return e;
}

tg_status phase2_run(const P2Input& in, void* scratch, size_t scratch_cap, P2Output& out,
                     const std::function<void*(size_t)>& fallback_table, cudaStream_t st, cudaEvent_t ev_keys,
                     int* launches, std::string& err, const P2Overlap& ov) {
    const P2Plan L = make_plan(in);
    const int W = in.W;
    Carve c{static_cast<uint8_t*>(scratch), 0, scratch_cap, true};
    const P2Regions R = carve(c, in, L);
    if (!c.ok) { err = "phase-2 scratch too small"; return TG_ERR_OOM; }

    P2_CK(setup(in, R, st), "k_setup");
    ++*launches;
    // counts per bin -> k-mers and packed records before each bin (of this run's bins)
    P2_CK(launch_bin_scan(in.binhist + in.bin_lo, in.bin_hi - in.bin_lo, R.kofs + in.bin_lo, R.rofs + in.bin_lo,
                          R.sums, st, launches),
          "scan");
    if (!in.deferred && in.n_kmers >> 32) {
        unsigned long long sum = 0;
        P2_CK(read_counters(ov, {R.kofs + in.bin_hi, 1}, {}, {}, &sum, st), "scan");
        if (!kmers_per_bin_ok(sum, in.n_kmers)) { err = bin_too_large(); return TG_ERR_UNSUPPORTED; }
    }

    KeysParams K{};
    K.packed = in.packed;
    K.desc = in.desc;
    K.desc_cap = in.desc_cap;
    K.n_desc = in.n_desc;
    K.n_one = in.max_desc;
    K.kofs = R.kofs;
    K.rofs = R.rofs;
    K.gfirst = R.gfirst;
    K.segs = R.segs;
    K.n_segs = in.n_segs;
    K.target = group_target(in);
    K.store = W == 1 ? CountShape<1>::CAP : CountShape<2>::CAP;
    K.k = in.k;
    K.recs = R.recs;
    K.groups[0] = R.normal;
    K.groups[1] = R.heavy;
    K.groups[2] = R.big;
    K.groups_cap = L.groups_cap;
    K.ctr = R.ctr;
    K.bin_lo = in.bin_lo;
    K.bin_hi = in.bin_hi;
    K.desc_sb = in.desc_sb;
    K.plan_split = plan_split(in);
    {
        const uint32_t warps = PLAN_THREADS / 32, n = in.n_segs * K.plan_split;
        k_plan<<<(n + warps - 1) / warps, PLAN_THREADS, 0, st>>>(K);  // before k_recs moves the cursors
    }
    P2_CK(cudaGetLastError(), "k_plan");
    ++*launches;
    if (in.n_lists && in.max_desc) {
        // A group's records land one 16 x W byte piece at a time at its cursor. With too
        // many groups open at once their partly written lines no longer stay in L2
        // until they are full, so jobs of many groups take several launches, each for
        // a share of the bins, although every launch reads all descriptors (603 M
        // records into 0.8 M groups: 1 launch 23.8 ms, 2 17.6, 4 16.7; 180 M records
        // into 0.23 M groups: 4.37, 4.53, 4.54).
        const uint32_t KP = 1 + (uint32_t)std::min<uint64_t>(7, in.n_kmers / group_target(in) >> 18);
        const uint32_t span = in.bin_hi - in.bin_lo;
        const dim3 grid((in.max_desc + RECS_PER_CTA - 1) / RECS_PER_CTA, in.n_lists);
        for (uint32_t kp = 0; kp < KP; ++kp) {
            KeysParams Kp = K;
            Kp.bin_lo = in.bin_lo + (uint32_t)((uint64_t)span * kp / KP);
            Kp.bin_hi = in.bin_lo + (uint32_t)((uint64_t)span * (kp + 1) / KP);
            if (W == 1) k_recs<1><<<grid, RECS_THREADS, 0, st>>>(Kp);
            else k_recs<2><<<grid, RECS_THREADS, 0, st>>>(Kp);
            P2_CK(cudaGetLastError(), "k_recs");
            ++*launches;
        }
    }
    if (ev_keys) P2_CK(cudaEventRecord(ev_keys, st), "event");

    CountParams Q{};
    Q.recs = R.recs;
    Q.k = in.k;
    Q.fallback = R.fb;
    Q.fallback_cap = FALLBACK_CAP;
    Q.ci = in.ci;
    Q.cx = in.cx;
    Q.out_keys = out.keys;
    Q.out_counts = out.counts;
    Q.out_sample = out.samples;
    Q.sample_tot = out.samples ? R.stot : nullptr;
    if (out.samples) P2_CK(cudaMemsetAsync(R.stot, 0, 4 * (size_t)in.n_samples, st), "memset");
    Q.out_cap = out.cap;
    Q.ctr = R.ctr;
    Q.retry_cap = L.retry_cap;
    const size_t sm = W == 1 ? sizeof(CountSmem<1>) : sizeof(CountSmem<2>);
    P2_CK(W == 1 ? set_smem_cap(k_count<1>, sm) : set_smem_cap(k_count<2>, sm), "smem");
    unsigned long long h[P2C_COUNT] = {};
    auto lists_ok = [&] {
        return h[P2C_NORMAL] <= L.groups_cap && h[P2C_HEAVY] <= L.groups_cap && h[P2C_BIG] <= L.groups_cap;
    };
    if (!in.deferred) {  // the groups: their number is known once k_plan has run
        P2_CK(read_counters(ov, {R.ctr, P2C_COUNT}, {}, {}, h, st), "phase 2");
        if (!lists_ok()) { err = "group list overflow"; return TG_ERR_TABLE; }
    }
    const unsigned long long ngroups = h[P2C_NORMAL];
    const unsigned cgrid = in.n_sm * COUNT_PER_SM;
    auto rounds = [&](const Group* list, unsigned long long n) -> cudaError_t {
        Q.list = list;
        Q.g_begin = 0;
        Q.g_end = n;
        const unsigned grid = (unsigned)std::min<unsigned long long>(n, R.split ? split_ctas(in) : cgrid);
        if (!grid) return cudaSuccess;
        cudaError_t e = W == 1 ? set_smem_cap(k_rounds<1>, sm) : set_smem_cap(k_rounds<2>, sm);
        if (e == cudaSuccess) e = cudaMemsetAsync(R.work + 16, 0, 8, st);
        if (e != cudaSuccess) return e;
        Q.work = R.work + 16;
        if (W == 1) k_rounds<1><<<grid, COUNT_THREADS, sm, st>>>(Q);
        else k_rounds<2><<<grid, COUNT_THREADS, sm, st>>>(Q);
        ++*launches;
        return cudaGetLastError();
    };
    // a global table with room for n keys: count() launches what fills it, then its pairs are written
    auto in_table = [&](uint64_t n, uint32_t sample, const std::function<cudaError_t(const FallbackParams&)>& count,
                        bool may_lack_room) -> tg_status {
        const uint64_t S = table_slots(n, in.k);
        if (!S) {
            if (!may_lack_room) err = "fallback table too large";
            return TG_ERR_TABLE;
        }
        const size_t kbytes = (size_t)S * key_bytes(W);
        const size_t bytes = kbytes + (size_t)S * 4 + 16;
        uint8_t* tab = may_lack_room && bytes > in.table_room ? nullptr : static_cast<uint8_t*>(fallback_table(bytes));
        if (!tab) {
            if (!may_lack_room) err = "no room for the fallback table";
            return TG_ERR_OOM;
        }
        FallbackParams F{};
        F.recs = R.recs;
        F.k = in.k;
        F.tkeys = tab;
        F.tcnt = reinterpret_cast<uint32_t*>(tab + kbytes);
        F.mask = (uint32_t)(S - 1);
        F.fail = reinterpret_cast<uint32_t*>(tab + kbytes + (size_t)S * 4);
        P2_CK(cudaMemsetAsync(F.fail, 0, 4, st), "memset");
        const unsigned grid = (unsigned)std::min<uint64_t>((S + 255) / 256, (uint64_t)in.n_sm * 8);
        if (W == 1) k_fb_init<1><<<grid, 256, 0, st>>>(F.tkeys, F.tcnt, S);
        else k_fb_init<2><<<grid, 256, 0, st>>>(F.tkeys, F.tcnt, S);
        P2_CK(count(F), "fallback");
        if (W == 1) k_fb_extract<1><<<grid, 256, 0, st>>>(F.tkeys, F.tcnt, S, Q, sample);
        else k_fb_extract<2><<<grid, 256, 0, st>>>(F.tkeys, F.tcnt, S, Q, sample);
        P2_CK(cudaGetLastError(), "fallback");
        *launches += 3;
        uint32_t failed = 0;
        P2_CK(cudaMemcpyAsync(&failed, F.fail, 4, cudaMemcpyDeviceToHost, st), "d2h");
        P2_CK(cudaStreamSynchronize(st), "fallback");
        if (failed) { err = "fallback table overflow"; return TG_ERR_TABLE; }
        return TG_OK;
    };
    Q.split = R.split;
    Q.retry = R.retry[0];
    Q.n_retry = R.aux;
    // ---- the largest groups, some of a sample to a table (of few MB for a group of a
    // million k-mers; without room for it, they are counted like the other large ones)
    uint64_t n_big = 0;
    auto count_big = [&]() -> tg_status {
        if (!h[P2C_BIG]) return TG_OK;
        std::vector<Group> big(h[P2C_BIG]);
        P2_CK(cudaMemcpyAsync(big.data(), R.big, big.size() * sizeof(Group), cudaMemcpyDeviceToHost, st), "d2h");
        P2_CK(cudaStreamSynchronize(st), "d2h");
        std::sort(big.begin(), big.end(), [](const Group& a, const Group& b) { return a.sample < b.sample; });
        P2_CK(cudaMemcpyAsync(R.big, big.data(), big.size() * sizeof(Group), cudaMemcpyHostToDevice, st), "h2d");
        P2_CK(W == 1 ? set_smem_cap(k_big<1>, sm) : set_smem_cap(k_big<2>, sm), "smem");
        for (size_t a = 0; a < big.size();) {
            size_t b = a;
            uint64_t nk = 0, most = 0;
            while (b < big.size() && big[b].sample == big[a].sample && b - a < 32768 &&
                   (b == a || nk + big[b].keys <= BIG_TABLE_KEYS)) {
                nk += big[b].keys;
                most = std::max<uint64_t>(most, big[b].hi - big[b].lo);
                ++b;
            }
            const dim3 grid((unsigned)std::min<uint64_t>((most + BIG_CHUNK - 1) / BIG_CHUNK, cgrid), (unsigned)(b - a));
            const tg_status s = in_table(nk, big[a].sample, [&](const FallbackParams& F) {
                Q.list = R.big;
                Q.g_begin = a;
                if (W == 1) k_big<1><<<grid, COUNT_THREADS, sm, st>>>(Q, F);
                else k_big<2><<<grid, COUNT_THREADS, sm, st>>>(Q, F);
                return cudaGetLastError();
            }, true);
            if (s == TG_OK) n_big += b - a;
            else if (s != TG_ERR_OOM && !(s == TG_ERR_TABLE && err.empty())) return s;
            else P2_CK(rounds(R.big + a, b - a), "k_rounds");
            a = b;
        }
        return TG_OK;
    };
    // ---- the others first, in `waves` launches over slices of their list; each slice's output
    // range goes to on_range as soon as it is final
    // (at least WAVE_KEYS k-mers each: a launch, and what it waits for, costs about 15 us)
    const uint32_t waves = ov.on_range && ov.wave_out && ov.wave_ev && !in.deferred
                               ? (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>({ov.waves, 16u, in.n_kmers / WAVE_KEYS})) : 1;
    uint64_t done = 0;  // output keys already handed to on_range
    // the first and the last wave are half as long as the others: nothing is copied
    // before the first, and nothing counted while the last one's pairs are
    auto wave_at = [&](uint32_t w) -> unsigned long long {
        if (w == 0 || w >= waves) return w ? ngroups : 0;
        return ngroups * (2 * w - 1) / (2 * (waves - 1));
    };
    for (uint32_t wv = 0; wv < waves; ++wv) {
        Q.list = R.normal;
        Q.n_list = in.deferred ? R.ctr + P2C_NORMAL : nullptr;
        Q.g_begin = wave_at(wv);
        Q.g_end = in.deferred ? L.groups_cap : wave_at(wv + 1);
        Q.work = R.work + wv;
        if (Q.g_end > Q.g_begin) {
            const unsigned grid = (unsigned)std::min<uint64_t>(cgrid, Q.g_end - Q.g_begin);
            if (W == 1) k_count<1><<<grid, COUNT_THREADS, sm, st>>>(Q);
            else k_count<2><<<grid, COUNT_THREADS, sm, st>>>(Q);
            P2_CK(cudaGetLastError(), "k_count");
            ++*launches;
        }
        if (waves > 1) {
            if (ov.wave_out_dev) k_peek<<<1, 32, 0, st>>>({R.ctr + P2C_OUT, 1}, {}, {}, ov.wave_out_dev + wv);
            else P2_CK(cudaMemcpyAsync(ov.wave_out + wv, R.ctr + P2C_OUT, 8, cudaMemcpyDeviceToHost, st), "d2h");
            P2_CK(cudaEventRecord(ov.wave_ev[wv], st), "event");
        }
    }
    Q.n_list = nullptr;
    // the large groups behind them, counted while the waves' pairs are copied
    if (!in.deferred) P2_CK(rounds(R.heavy, h[P2C_HEAVY]), "k_rounds");
    if (waves > 1) {
        for (uint32_t wv = 0; wv < waves; ++wv) {
            P2_CK(cudaEventSynchronize(ov.wave_ev[wv]), "wave");
            const uint64_t hi = std::min<uint64_t>(*(const volatile unsigned long long*)(ov.wave_out + wv), out.cap);
            if (hi > done) {
                const tg_status rs = ov.on_range(done, hi);
                if (rs != TG_OK) { err = "result copy failed"; return rs; }
                done = hi;
            }
        }
    }
    if (!in.deferred) {
        const tg_status s = count_big();
        if (s != TG_OK) return s;
    }
    // ---- groups that came back as key-hash parts: pass p reads retry[p & 1], writes the other
    for (int pass = 0;; ++pass) {
        unsigned long long hr[1 + P2C_COUNT + 8];
        P2_CK(read_counters(ov, {R.aux + (pass & 1), 1}, {R.ctr, P2C_COUNT},
                            {in.read_back, pass == 0 ? std::min(in.n_read, 8u) : 0}, hr, st), "phase 2");
        unsigned long long nret = hr[0];
        for (int c = 0; c < P2C_COUNT; ++c) h[c] = hr[c + 1];
        if (pass == 0) {
            for (uint32_t c = 0; c < std::min(in.n_read, 8u); ++c) out.read_back[c] = hr[1 + P2C_COUNT + c];
            if (in.deferred) {
                if (!lists_ok()) { err = "group list overflow"; return TG_ERR_TABLE; }
                if (h[P2C_BIG] || h[P2C_HEAVY]) {  // larger groups, rare in a small job, counted now
                    const tg_status s = count_big();
                    if (s != TG_OK) return s;
                    P2_CK(rounds(R.heavy, h[P2C_HEAVY]), "k_rounds");
                    P2_CK(read_counters(ov, {R.aux, 1}, {R.ctr, P2C_COUNT}, {}, hr, st), "phase 2");
                    nret = hr[0];
                    for (int c = 0; c < P2C_COUNT; ++c) h[c] = hr[c + 1];
                }
            }
        }
        if (nret > L.retry_cap) { err = "too many groups to split"; return TG_ERR_TABLE; }
        if (nret == 0) break;
        Q.retry = R.retry[(pass + 1) & 1];
        Q.n_retry = R.aux + ((pass + 1) & 1);
        P2_CK(cudaMemsetAsync(Q.n_retry, 0, 8, st), "memset");
        P2_CK(rounds(R.retry[pass & 1], nret), "k_rounds");
    }
    out.fallback_groups = h[P2C_FALLBACK] + n_big;
    // ---- key ranges that did not fit in shared memory
    if (h[P2C_FALLBACK] > 0) {
        if (h[P2C_FALLBACK] > FALLBACK_CAP) { err = "too many overflowing groups"; return TG_ERR_TABLE; }
        std::vector<Group> fl(h[P2C_FALLBACK]);
        P2_CK(cudaMemcpyAsync(fl.data(), R.fb, fl.size() * sizeof(Group), cudaMemcpyDeviceToHost, st), "d2h");
        P2_CK(cudaStreamSynchronize(st), "d2h");
        for (const Group& g : fl) {
            const tg_status s = in_table(g.keys, g.sample, [&](FallbackParams F) {
                F.lo = g.lo;
                F.hi = g.hi;
                F.parts = g.parts;
                F.part = g.part;
                const unsigned grid = (unsigned)in.n_sm * 4;
                if (W == 1) k_fb_insert<1><<<grid, 256, 0, st>>>(F);
                else k_fb_insert<2><<<grid, 256, 0, st>>>(F);
                return cudaGetLastError();
            }, false);
            if (s != TG_OK) return s;
        }
        P2_CK(read_counters(ov, {R.ctr, P2C_COUNT}, {}, {}, h, st), "fallback");
    }
    out.n_out = h[P2C_OUT];
    if (ov.on_range && std::min<uint64_t>(out.n_out, out.cap) > done) {
        const tg_status rs = ov.on_range(done, std::min<uint64_t>(out.n_out, out.cap));
        if (rs != TG_OK) { err = "result copy failed"; return rs; }
    }
    out.distinct = h[P2C_DISTINCT];
    if (out.samples && out.n_samples > 1 && out.n_samples <= in.n_samples && out.keys2 && out.counts2 && out.sample_off) {
        // sample-major copy: the scan of the samples' totals, the scatter
        const uint64_t n = std::min<uint64_t>(out.n_out, out.cap);
        const unsigned grid = (unsigned)in.n_sm * 8;
        P2_CK(launch_scan(R.stot, out.n_samples, out.sample_off, R.sums, st, launches), "scan");
        unsigned long long* cur = R.scur;  // the offsets, copied, as cursors
        P2_CK(cudaMemcpyAsync(cur, out.sample_off, 8 * (size_t)out.n_samples, cudaMemcpyDeviceToDevice, st), "copy");
        if (out.reorder_after) P2_CK(cudaStreamWaitEvent(st, out.reorder_after, 0), "wait");
        if (W == 1) k_samp_scatter<1><<<grid, 256, 0, st>>>(out.keys, out.counts, out.samples, n, cur, out.keys2, out.counts2);
        else k_samp_scatter<2><<<grid, 256, 0, st>>>(out.keys, out.counts, out.samples, n, cur, out.keys2, out.counts2);
        P2_CK(cudaGetLastError(), "k_samp_scatter");
        *launches += 1;
        P2_CK(cudaStreamSynchronize(st), "sample order");
    }
    out.groups = h[P2C_NORMAL] + h[P2C_HEAVY] + h[P2C_BIG];
    out.heavy_groups = h[P2C_HEAVY] + h[P2C_BIG];
    if (out.n_out > out.cap) { err = "output capacity exceeded"; return TG_ERR_TABLE; }
    return TG_OK;
}

}  // namespace tg
