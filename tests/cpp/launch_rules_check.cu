// Host rules of the launch headers, checked against their definitions. Host
// code only: nvcc compiles it for sm_100a, but nothing runs on a GPU.
#include <chrono>
#include <cstdio>

#include "zlfft_istft.cuh"

using namespace zlfft;

static int bad = 0;
static void expect(bool ok, const char* what) {
    if (!ok) {
        ++bad;
        printf("FAILED: %s\n", what);
    }
}

// The run length by trying every one: the cheapest between the shortest that
// takes one wave of groups and 4 (K - 1), the shortest of equals.
static long long run_by_trying(long long blocks, int k, long long sms, int groups) {
    const long long cap = sms * groups, rmin = (blocks + cap - 1) / cap;
    long long run = rmin, best = -1;
    for (long long r = rmin; r <= 4LL * (k - 1); ++r) {
        const long long g = ((blocks + r - 1) / r + sms - 1) / sms;
        const long long cost = (r + k - 1) * (2 * g > 3 ? 2 * g : 3);
        if (best < 0 || cost < best) best = cost, run = r;
    }
    return run;
}

int main() {
    // two transforms per thread: never while one wave of one per thread holds
    // the batch, always over many waves; on a smaller or larger GPU too
    for (int sms : {148, 132, 64, 16}) {
        const long long cap1 = 5LL * sms, cap2 = 4LL * sms;
        for (long long t = 1; t <= cap1; ++t) expect(!pair_pays(t, cap1, cap2), "one wave: one transform per thread");
        for (long long t = cap1 + 1; t <= 2 * cap2; ++t) expect(pair_pays(t, cap1, cap2), "one wave of pairs against two");
        for (long long t = 2 * cap2 + 1; t <= 2 * cap1; ++t) expect(!pair_pays(t, cap1, cap2), "two waves against two of pairs");
        for (long long t = 8 * cap2 + 1; t <= 40 * cap2; t += 7) expect(pair_pays(t, cap1, cap2), "many waves: pairs");
    }
    printf("pairs: %s\n", bad ? "bad" : "ok");
    // launches that begin when the one before is done: short tiles in the second
    // of two waves, passes of one to four waves whose last is under half full;
    // none beside other launches of the call
    const LaunchCtx alone{148, nullptr, false}, beside{148, nullptr, true};
    for (long long cap : {148LL, 444LL, 740LL}) {
        for (long long n = 1; n <= 6 * cap; ++n) {
            expect(tile_overlaps(alone, 8, n, cap) == !(n > cap && n < 2 * cap), "short tiles");
            expect(tile_overlaps(alone, 9, n, cap) && tile_overlaps(beside, 8, n, cap), "other tiles");
            const bool ragged = n > cap && n < 4 * cap && n % cap != 0 && n % cap < (cap + 1) / 2;
            expect(pass_overlaps(alone, n, cap) == !ragged, "passes");
            expect(pass_overlaps(beside, n, cap), "passes of two chunks");
        }
    }
    // shared memory asked for: the even share of CTAs fits an SM and one more
    // does not, where more would fit, but two even shares would not
    for (int per_sm = 1; per_sm <= 24; ++per_sm) {
        const size_t own = kSmemPerSm / per_sm / 1024 * 1024 - kSmemReserve;
        for (long long grid = 1; grid <= 148LL * per_sm; ++grid) {
            const int k = (int)((grid + 147) / 148);
            const size_t got = balanced_smem(alone, grid, per_sm, own);
            const size_t each = got + kSmemReserve;
            if (k < per_sm && 2 * k > per_sm)
                expect(each % 1024 == 0 && k * each <= kSmemPerSm && (2 * k) * each > kSmemPerSm && got <= kSmemPerCta, "share");
            else
                expect(got == own, "own size");
            expect(balanced_smem(beside, grid, per_sm, own) == own, "own size beside others");
        }
    }
    printf("launches: %s\n", bad ? "bad" : "ok");
    // inverse STFT: the weighed runs give what trying every length gives
    for (int k : {1, 2, 3, 4, 8, 16, 64, 512, 8192})
        for (int groups : {1, 2, 5, 10, 15, 32})
            for (long long sms : {148LL, 64LL})
                for (long long blocks = 1; blocks < 4000000; blocks = blocks * 5 / 3 + 1)
                    expect(istft_run(blocks, k, sms, groups) == run_by_trying(blocks, k, sms, groups), "run length");
    // and take no longer for many overlapping frames than for few
    long long sum = 0;
    const auto t0 = std::chrono::steady_clock::now();
    for (int i = 0; i < 20000; ++i) sum += istft_run(9000 + i, 8192, 148, 15);
    const double us = std::chrono::duration<double, std::micro>(std::chrono::steady_clock::now() - t0).count() / 20000;
    expect(us < 10 && sum > 0, "host time of the run length");
    printf("runs: %s\n", bad ? "bad" : "ok");
    // CTAs of one group: one wave of single frames, on SMs that hold several groups
    for (int groups = 1; groups <= 21; ++groups) {
        expect(istft_has_single(groups) == (groups >= 4), "sizes with single groups");
        const long long slots = 148LL * groups;
        for (long long runs : {1LL, 2LL, slots - 1, slots}) {
            expect(istft_single(runs, 1, slots), "a wave of single frames");
            expect(!istft_single(runs, 2, slots), "several frames a group");
        }
        expect(!istft_single(slots + 1, 1, slots), "more than a wave");
    }
    printf("single: %s\n", bad ? "bad" : "ok");
    return bad ? 1 : 0;
}
