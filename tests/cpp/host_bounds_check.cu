// host_bounds_check.cu — bounds that the host code relies on where a run's buffers
// are sized before its counts are known, checked without a GPU.
#include <algorithm>
#include <cstdio>

#include "tg_launch.h"

using namespace tg;

static int fails = 0;
#define CHECK(cond, ...)                                           \
    do {                                                           \
        if (!(cond)) {                                             \
            if (++fails <= 20) {                                   \
                std::printf("FAIL line %d: ", __LINE__);           \
                std::printf(__VA_ARGS__);                          \
                std::printf("\n");                                 \
            }                                                      \
        }                                                          \
    } while (0)

// Records of the first list when every position of its chunk starts one and the last
// of them is a chain to the stream's end, split every L positions.
static void check_cut_lists() {
    for (int k = 2; k <= 63; ++k)
        for (int m = 1; m < k && m <= 32; ++m)
            for (uint64_t n : {1ull, 1000ull, 524288ull, 3000000ull, 4194304ull, 4600000ull, 3100000000ull}) {
                const uint32_t L = 256 - (uint32_t)k;
                const uint64_t chunk = cut_layout(k - m, k, 1, false, n, 152).chunk;
                const uint64_t in_chunk = std::min(chunk, n), behind = n - in_chunk;
                const uint64_t most = cut_list_most(chunk, n, L);
                CHECK(most >= in_chunk + (behind + L - 1) / L, "k=%d m=%d n=%llu: a list of %llu", k, m,
                      (unsigned long long)n, (unsigned long long)most);
                CHECK(most <= chunk + n / L + 64, "k=%d m=%d n=%llu: a list of %llu", k, m, (unsigned long long)n,
                      (unsigned long long)most);
            }
}

// A global table's slots against its k-mers, and the probes that a mask of 32 bits allows.
static void check_tables() {
    for (int k : {16, 31, 32, 63})
        for (uint64_t n : {0ull, 1ull, 511ull, 65537ull, (1ull << 30) - 1, 1ull << 30, (1ull << 31) - 1}) {
            const uint64_t S = table_slots(n, k);
            CHECK(S >= 2 * n + 1 && S <= 1ull << 32 && (S & (S - 1)) == 0, "%llu slots for %llu k-mers",
                  (unsigned long long)S, (unsigned long long)n);
            CHECK((uint32_t)(S - 1) > n, "%u probes among %llu k-mers", (uint32_t)(S - 1), (unsigned long long)n);
        }
    for (uint64_t n : {1ull << 31, 1ull << 32, 1ull << 40}) CHECK(table_slots(n, 31) == 0, "no table");
    // few k-mers differ, however many there are
    CHECK(table_slots(1ull << 40, 9) >= 2ull << 18 && table_slots(1ull << 40, 9) <= 4ull << 18, "4^9 k-mers");
    CHECK(table_slots(1ull << 40, 2) == 1024 && table_slots(100, 9) == 1024, "small tables");
}

// Bin counts as the cut adds them up, records of 225 k-mers in 15 pieces: the sum tells
// a bin of 2^32 k-mers or more.
static void check_bin_counts() {
    for (uint64_t in_one : {(1ull << 32) / 225 - 1, (1ull << 32) / 225 + 1, (3ull << 32) / 225 + 7}) {
        uint64_t hist[2] = {0, 0}, kmers = 0, sum = 0;
        for (uint64_t r = 0; r < in_one + 1000; ++r, kmers += 225)
            hist[r >= in_one] += ((uint64_t)rec_pieces(225) << 32) | 225;
        for (uint64_t h : hist) sum += h & 0xFFFFFFFFull;
        CHECK(kmers_per_bin_ok(sum, kmers) == (in_one * 225 < 1ull << 32), "%llu k-mers of one bin",
              (unsigned long long)in_one * 225);
    }
}

// The group sizes of a tuned context: all different, the default's the largest.
static void check_group_sizes() {
    for (int W = 1; W <= 2; ++W) {
        uint32_t before = 0;
        for (uint32_t pct : TUNE_PCT) {
            CHECK(group_keys(W, pct) > before, "%u %% gives %u k-mers again (W=%d)", pct, group_keys(W, pct), W);
            before = group_keys(W, pct);
        }
        CHECK(before == group_keys(W, P2Input{}.group_pct) && before == group_keys(W, 100), "W=%d: %u", W, before);
    }
}

int main() {
    check_cut_lists();
    check_group_sizes();
    check_tables();
    check_bin_counts();
    if (fails) {
        std::printf("%d checks failed\n", fails);
        return 1;
    }
    std::printf("OK\n");
    return 0;
}
