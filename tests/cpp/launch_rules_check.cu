// Host rules of the launch headers, checked against their definitions. Host
// code only: nvcc compiles it for sm_100a, but nothing runs on a GPU.
#include <cstdio>

#include "zlfft_launch.cuh"

using namespace zlfft;

static int bad = 0;
static void expect(bool ok, const char* what) {
    if (!ok) {
        ++bad;
        printf("FAILED: %s\n", what);
    }
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
    return bad ? 1 : 0;
}
