// Host check of the rule by which the mixed kernel takes a wave's candidate
// pairs in parts (wave_part): the parts cover the warps in order, and a part's
// pairs, with the 32 that each warp may add to the cursor past the end, fit an
// int.  And of where a tet's pairs start among 32 (start_bit).  Built for the
// host only, with the compiler's check for undefined behaviour where it has
// one; no GPU.
#include "../adeco_gb300/csrc/kernels.cuh"

#include <climits>
#include <cstdio>
#include <random>

using namespace adeco;

static long bad = 0;

static int parts_of(const int pairs[kWarps])
{
    int n = 0;
    for (int first = 0; first < kWarps; ++n) {
        int total = -1;
        const int end = wave_part(pairs, first, total);
        long long sum = 0;
        for (int w = first; w < end; ++w) sum += pairs[w];
        // more than the part could not be taken: the next warp's pairs do not fit
        const bool most = end == kWarps || sum + pairs[end] + 32LL * kWarps > INT_MAX;
        if (end <= first || end > kWarps || sum != total || sum + 32LL * kWarps > INT_MAX || !most) {
            ++bad;
            return n;
        }
        first = end;
    }
    return n;
}

int main()
{
    const int most = (int)(32 * kMaxPairsPerTet);  // a warp's tets
    int full[kWarps], none[kWarps], edge[kWarps], over[kWarps];
    for (int w = 0; w < kWarps; ++w) {
        full[w] = most;
        none[w] = 0;
        edge[w] = over[w] = kMaxPartPairs / kWarps;
    }
    edge[kWarps - 1] = kMaxPartPairs - (kWarps - 1) * edge[0];
    over[kWarps - 1] = edge[kWarps - 1] + 1;
    bad += parts_of(full) != kWarps;  // two of 2^30 pairs are already 2^31
    bad += parts_of(none) != 1;
    bad += parts_of(edge) != 1;
    bad += parts_of(over) != 2;
    std::mt19937_64 rng(5);
    for (int i = 0; i < 200000; ++i) {
        int pairs[kWarps];
        for (int w = 0; w < kWarps; ++w) pairs[w] = (int)(rng() % (unsigned)(most + 1)) >> (rng() % 31);
        parts_of(pairs);
    }
    // a tet's start among the 32 pairs that a warp takes, against 64-bit arithmetic
    const int rels[] = {0, 1, 31, 32, 1 << 20, (1 << 30) - 1, 1 << 30};
    for (int rel : rels)
        for (int skip = 0; skip < 32; ++skip) {
            const long long starts[] = {0, 1, rel - 1LL, rel, rel + 1LL, rel + 31LL - skip, rel + 32LL - skip, rel + 33LL,
                                        (1LL << 30) - 1, INT_MAX - 1LL, INT_MAX};
            for (long long start : starts) {
                if (start < 0) continue;
                const long long at = start - rel + skip;
                const unsigned want = start > rel && at < 32 ? 1u << at : 0u;
                bad += start_bit((int)start, rel, skip) != want;
            }
        }
    std::printf("parts of a wave: %s (%ld)\n", bad ? "FAIL" : "ok", bad);
    return bad ? 1 : 0;
}
