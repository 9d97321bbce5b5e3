// tg_launch.h — host-side launchers of the counting kernels (defined in
// tg_phase1.cu, tg_phase2.cu, tg_api.cu) shared by the entry points.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <functional>
#include <string>
#include <vector>

#include "tuna_gpu.h"

#include "tg_internal.cuh"

namespace tg {
// A job of at most this many stream bytes runs in one go: buffers sized by bounds, the
// counts read on the device, one wait at the end (P2Input::deferred).
constexpr uint64_t DEFER_BYTES = 4u << 20;
// Shapes of the cut; seg: k-mer start positions per thread and tile (cut_layout).
size_t cut_smem_bytes(int w, int k, uint32_t p1, bool exp, int seg = 128);
uint64_t cut_tile(int w, bool exp, int seg = 128);  // k-mer start positions per tile of a cut CTA
uint32_t cut_ctas_per_sm(int w, int k, uint32_t p1, bool exp, int seg = 128);
CutLayout cut_layout(int w, int k, uint32_t p1, bool exp, uint64_t n, uint32_t n_sm);
// The most records that one list of a cut of n positions can get (L: CutParams::L): one
// per position of its chunk, and the forced splits, L positions apart, of the chain
// that is open at the chunk's end, wherever that ends (a homopolymer's: the whole stream).
uint64_t cut_list_most(uint64_t chunk, uint64_t n, uint32_t L);
cudaError_t launch_prepare(const PrepareParams& P, cudaStream_t st);
// Packed words (a multiple of 4) for a stream of n bytes, padding included.
uint64_t packed_words_for(uint64_t n);
// Packs what of the stream is there and was not at the launch before; most: an
// upper bound of its length.
cudaError_t launch_pack(const uint8_t* seq, const Avail& av, uint64_t most, uint32_t* packed, uint32_t* valid,
                        unsigned long long* n_bases, int n_sm, cudaStream_t st);
cudaError_t launch_cut(const CutParams& P, const HashTables* gT, bool exp, cudaStream_t st);
// Exclusive scans of n >= 1 counts into n + 1 entries (the last: the total, which
// goes to *total too if given); scratch holds scan_scratch(n) u64, 16-byte aligned.
uint64_t scan_scratch(uint64_t n);
cudaError_t launch_scan(const uint32_t* in, uint64_t n, unsigned long long* out, unsigned long long* scratch,
                        cudaStream_t st, int* launches, unsigned long long* total = nullptr);
cudaError_t launch_bin_scan(const unsigned long long* hist, uint64_t n, unsigned long long* kofs,
                            unsigned long long* rofs, unsigned long long* scratch, cudaStream_t st, int* launches);
// FASTA/FASTQ lexing on the device (tg_lex.cu). raw must be 16-byte aligned;
// out receives at most len bytes. Totals are written to device memory (*dtot,
// inside scratch) and are valid once the stream reaches them.
struct LexTotals {
    unsigned long long out;        // stream bytes written
    unsigned long long drop_from;  // FASTQ: bytes from here on were not emitted (end-of-file rule)
    uint32_t final_state;          // automaton state at the end of the file
    long long last_na;             // FASTQ: 1 + offset of the last non-ACGT byte so far, 0: none
    uint32_t irregular;            // bit 0: FASTQ with an empty header line at offset 63 mod 64 (parse
                                   // on the host); bit 1: a staging wait timed out (device error)
};
size_t lex_scratch_bytes(uint64_t len);
// A file may be lexed in pieces, in order, while the rest of it is still copied:
// bytes [lo, hi) of it, lo a multiple of LEX_PIECE_UNIT and hi too or len.
constexpr uint64_t LEX_PIECE_UNIT = 16384;
cudaError_t launch_lex(const uint8_t* raw, uint64_t len, bool fastq, uint8_t* out, void* scratch, int n_sm,
                       cudaStream_t st, LexTotals** dtot, int* launches, uint64_t lo, uint64_t hi,
                       unsigned long long* piece_out = nullptr);  // receives the stream's length so far
// Output formatting on the device (tg_format.cu): n pairs to the bytes of
// format fmt (tg_format). TSV writes its byte count to d_total (device-
// writable, e.g. mapped host memory); KFF and RAW records have a fixed size,
// fmt_max_bytes, and leave d_total alone.
size_t fmt_scratch_bytes(uint64_t n_pairs);
uint64_t fmt_max_bytes(int fmt, int k, uint64_t n_pairs);
cudaError_t launch_format(int fmt, int k, const uint64_t* keys, const uint32_t* counts, uint64_t n, uint8_t* out,
                          void* scratch, int n_sm, cudaStream_t st, unsigned long long* d_total, int* launches);
// Digest of n pairs (tg_job_result_digest) into out[4] (device): pairs, count
// sum, h1, h2.
cudaError_t launch_digest(int k, const uint64_t* keys, const uint32_t* counts, uint64_t n, unsigned long long* out,
                          int n_sm, cudaStream_t st, int* launches);
// A copy between device memory and host memory (tg_link.cu): done by a kernel
// through the mapped address when the host side is page-locked memory mapped
// for the current device (and both sides are equally aligned mod 16), else by
// cudaMemcpyAsync; ordered on st like cudaMemcpyAsync.
cudaError_t link_copy(void* dst, const void* src, size_t bytes, cudaMemcpyKind kind, cudaStream_t st, int n_sm,
                      int* launches = nullptr);
// Many copies from mapped host memory in one launch (a copy of its own for each of
// 400 samples of half a megabyte ran at 120 GB/s of the link's 200): piece q is len
// bytes from src to dst, equally aligned mod 16, then `fill` (at most 32) line feeds.
struct LinkPiece {
    const uint8_t* src;
    uint8_t* dst;
    uint32_t len, fill;
};
constexpr uint32_t LINK_PIECE = 32u << 10;  // bytes per piece, a multiple of 16; small: 38 CTAs share 13 MB evenly
cudaError_t link_gather(const LinkPiece* pieces, uint32_t n, cudaStream_t st, int ctas, int* launches = nullptr);
// The device address of host memory that is page-locked and mapped for the
// current device, else null (pageable memory, device memory, bad pointers).
const void* mapped_address(const void* host);
// Spill mode (tg_spill.cu): records of the phase-1 descriptor lists to
// per-bucket staging areas (bucket = bin >> shift, at most SPILL_MAX_BUCKETS).
// launch_spill_size: totals[b] records and totals[nb + b] bytes of bucket b.
// launch_spill_write: cursors[b] / cursors[nb + b] start at bucket b's staging
// base (records / bytes); host_shift[b] = the bucket stream's length before
// this chunk minus its staging byte base; staging byte bases and stream lengths
// are multiples of 4. launch_rebase: add `add` to the start of n descriptors.
constexpr uint32_t SPILL_MAX_BUCKETS = 1024;
cudaError_t launch_spill_size(const uint64_t* desc, uint64_t desc_cap, const uint32_t* n_desc, uint32_t n_lists,
                              int k, int shift, uint32_t nb, unsigned long long* totals, cudaStream_t st);
cudaError_t launch_spill_write(const uint32_t* packed, const uint64_t* desc, uint64_t desc_cap, const uint32_t* n_desc,
                               uint32_t n_lists, int k, int shift, uint32_t nb, unsigned long long* cursors,
                               const long long* host_shift, uint64_t* out_desc, uint8_t* out_bytes, cudaStream_t st);
cudaError_t launch_rebase(uint64_t* desc, uint64_t n, uint64_t add, int n_sm, cudaStream_t st);
size_t key_bytes(int W);
uint32_t count_slots(int W);  // the unit of P2Input::group_pct
// K-mers of a group that takes pct % of the unit: at most what a CTA's store holds
// (4,096 or, of two words, 3,072).
uint32_t group_keys(int W, uint32_t pct);
// The group sizes that a tuned context tries (TG_CTX_AUTOTUNE), the store's among them:
// 2,048, 2,867 and 4,096 or 3,072 k-mers (155 Mbp, k=31 m=21: 1.57, 1.42, 1.35 ms of counting).
constexpr uint32_t TUNE_PCT[] = {25, 35, 50};
// Slots of a table in global memory for n k-mers of length k, of which at most 4^k
// differ: a power of two, more than half of them free. 0: more than 2^32.
uint64_t table_slots(uint64_t n, int k);

// Whether no bin of a job of n_kmers k-mers, whose bins' k-mers add up to sum, holds
// 2^32 of them or more: each such bin is short by a multiple of 2^32.
inline bool kmers_per_bin_ok(uint64_t sum, uint64_t n_kmers) { return sum == n_kmers; }
inline const char* bin_too_large() { return "a bin holds more than 2^32 k-mers"; }

// Phase 2 of one job, shared by the entry points: the phase-1 descriptor lists
// and the k-mer counts per bin in, distinct keys and counts (and their
// samples) out.
// Bins of one sample per segment; the host helper below lays them out.
struct SampleBins {
    std::vector<unsigned long long> start;  // [n + 1] stream position of each sample, then the end
    std::vector<uint32_t> base;             // [n] first bin
    std::vector<uint8_t> bits;              // [n] log2 bins
    std::vector<Segment> segs;
};
// Shares 2^bin_bits bins out among samples in proportion to their length (a
// power of two each) and cuts each sample's bins into segments of at most
// seg_bins bins.
SampleBins layout_bins(const std::vector<unsigned long long>& sample_start, uint32_t seg_bins,
                       int bin_bits = BIN_BITS);
// log2 of the bins of a job of n stream bytes, n_samples samples and 2^seg_bits
// segments that shares its bins with no other run.
int job_bin_bits(uint64_t n, uint32_t n_samples, uint32_t seg_bits);
struct P2Input {
    int W, k;                          // key words, k
    const Segment* segs;               // [n_segs] (host): runs of bins of one sample, cut into groups
    uint32_t n_segs;
    uint32_t n_sm;
    const uint32_t* packed;
    const uint64_t* desc;              // [n_lists][desc_cap] phase-1 descriptors
    uint64_t desc_cap;
    uint32_t n_lists;
    const uint32_t* n_desc;            // [n_lists] descriptors per list (device); null: one list of max_desc
    uint32_t max_desc;                 // descriptors of the longest list
    const unsigned long long* binhist; // [all_bins] k-mers and packed records per bin (device)
    uint64_t n_kmers;                  // k-mer instances in all
    uint64_t n_recs;                   // packed records in all
    uint64_t ci, cx;
    bool roomy = false;                // scratch for splitting large groups may be taken
    uint64_t table_room = ~0ull;       // bytes that a table for the largest groups may take
    uint32_t n_samples = 1;
    // the bins counted by this run (all by default); segs must lie inside, and
    // n_kmers and n_recs count only theirs
    uint32_t bin_lo = 0, bin_hi = 1u << BIN_BITS;
    uint32_t all_bins = 1u << BIN_BITS;  // bins of the job
    int desc_sb = DESC_START_BITS;       // start bits of a descriptor
    uint32_t group_pct = 50;  // k-mers per group (group_keys)
    // Phase 1 may still run: n_kmers, n_recs and max_desc are upper bounds, the
    // counts are read on the device, and the host waits once, at the end; read_back
    // (n_read u64, device) then goes to P2Output::read_back.
    bool deferred = false;
    const unsigned long long* read_back = nullptr;
    uint32_t n_read = 0;
};
struct P2Output {
    void* keys;                        // u64 x W per distinct k-mer
    uint32_t* counts;
    uint32_t* samples = nullptr;       // sample of each pair, or null
    // jobs of several samples: the pairs again, sample-major, and the first pair
    // of each sample (n_samples + 1 entries, device)
    uint32_t n_samples = 1;
    void* keys2 = nullptr;
    uint32_t* counts2 = nullptr;
    unsigned long long* sample_off = nullptr;
    uint64_t cap;
    uint64_t n_out, distinct, groups, heavy_groups, fallback_groups;
    // the sample-major scatter waits for this event first (an earlier job's
    // copy of keys2/counts2 to the host may still be running), or null
    cudaEvent_t reorder_after = nullptr;
    unsigned long long read_back[8] = {};
};
// Results handed out while phase 2 still runs: the first counting pass runs in
// `waves` launches, and after each one on_range(lo, hi) is called (on the host,
// in order) with the output range [lo, hi) that is now final in P2Output;
// the last call comes after the retry passes. wave_out: pinned host memory of
// `waves` u64; wave_ev: `waves` events. Empty on_range: one launch, no calls.
struct P2Overlap {
    uint32_t waves = 1;
    unsigned long long* wave_out = nullptr;      // host address of mapped pinned memory, OVERLAP_WORDS u64
    unsigned long long* wave_out_dev = nullptr;  // its device address
    cudaEvent_t* wave_ev = nullptr;
    std::function<tg_status(uint64_t lo, uint64_t hi)> on_range;
};
// wave_out layout: [0, 16) output totals after each wave, [16, 64) counter reads.
// Counters are read back by a one-warp kernel storing into this mapped memory,
// not by cudaMemcpyAsync: a copy-engine read would queue behind the result
// copies already issued on the copy stream.
constexpr uint32_t OVERLAP_WORDS = 64;
// n u64 of device memory to mapped host memory (device address dst), by a kernel.
cudaError_t launch_peek(const unsigned long long* src, uint32_t n, unsigned long long* dst, cudaStream_t st);
// Device scratch one run needs (packed records included).
size_t phase2_scratch_bytes(const P2Input& in);
// Runs phase 2 on `st` and waits for it. fallback_table(bytes) returns device
// memory for a global table (or null); ev_keys (optional) is recorded once the
// packed records are written.
tg_status phase2_run(const P2Input& in, void* scratch, size_t scratch_cap, P2Output& out,
                     const std::function<void*(size_t)>& fallback_table, cudaStream_t st, cudaEvent_t ev_keys,
                     int* launches, std::string& err, const P2Overlap& ov = P2Overlap());

}  // namespace tg
