// Host check of the rule by which the mixed kernel takes a wave's candidate
// pairs in parts (wave_part): the parts cover the warps in order, and a part's
// pairs, with the 32 that each warp may add to the cursor past the end, fit an
// int.  Built for the host only; no GPU.
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
    std::printf("parts of a wave: %s (%ld)\n", bad ? "FAIL" : "ok", bad);
    return bad ? 1 : 0;
}
